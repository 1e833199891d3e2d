// Tensor-core (tcgen05) fused SDF field: hash-grid encoding + SDFNetwork MLP
// (models/fields.py:76-99) forward and backward, fp32-accurate (3xTF32).
//
// A CTA owns 128-point tiles (persistent over tiles) with 16 warps in the forward
// kernels and 32 in the backward ones: warp w serves TMEM lane quadrant q = w % 4
// (points 32q..32q+31 of the tile) as member g = w / 4 of that quadrant's group of
// four or eight.  The members split the per-point work -- hash-grid levels
// (interleaved, see level_of), hidden units -- and write their parts of each point's
// row straight into the point's TMEM lane, where the tensor core reads it as the A
// operand.  One to three threads issue the MMAs; everyone waits on an mbarrier
// (bounded).
//
// MLP input order inside the kernels (K = 40): encoding features first
// (level l, feature f -> column 2l + f), then x (columns 32..34), then zeros;
// W0 is permuted to match when it is staged, and the weight gradient is
// permuted back when it is flushed.
//
// Forward:  H = IN W0^T (TMEM), act = softplus(H + b0), out = W1 act + b1.
// Backward: recompute H, dH = (W1^T g) * softplus'(H + b0),
//           dIN = dH W0 (TMEM) -> table-gradient scatter (+ dL/dx),
//           dW0 += dH^T IN over the CTA's points (TMEM, A = [dH_hi; dH_lo]
//           stacked as 128 rows so two MMAs per K step give all four
//           hi/lo products), db0 from a row of ones in IN^T,
//           dW1 per point of the tile in TMEM (several outputs: by warp
//           reductions); db1 is a column sum of its own (field.cu).
#include "field_common.cuh"
#include "tc.cuh"

#include <cuda_bf16.h>

#include <string.h>

namespace sn {
namespace {

constexpr int kTile = 128;
constexpr int kK1 = 40;        // MLP input width inside the kernels (35 used)
constexpr int kN2 = 48;        // dIN columns (N of the second MMA; 35 used)
constexpr int kXCol = 32;      // first column of x in the permuted input
constexpr int kOnesRow = 35;   // row of ones in IN^T (gives db0)
constexpr uint32_t kCols = 256;      // forward: up to two CTAs per SM
constexpr uint32_t kBwdCols = 512;   // backward: one CTA per SM
// IN^T and [dH_hi; dH_lo] (K = the tile's points, written one point per
// thread): core matrices 144 bytes apart along K so a warp's 32 stores of one
// row fall in 32 banks.
constexpr uint32_t kLboP = 144, kSboP = (kTile / 4) * kLboP;

// The three 3xTF32 passes of a GEMM: the forward issues hi.hi and the two small
// products from threads of two warps into an accumulator each (no ordering between
// the threads is needed), summed by the readers; one mbarrier counts a commit per
// issuing thread.  The other kernels issue them from one thread into one
// accumulator, the small products first (mma_3x).
//
// Forward TMEM columns (256): H part 0 [0,64), parts 1+2 [64,128); input
// rows hi [128,168), lo [168,208).
constexpr uint32_t kFwdColH0 = 0, kFwdColH1 = 64, kFwdColInHi = 128, kFwdColInLo = 128 + kK1;
// Backward TMEM columns (512): H [0,64), dIN of even steps [64,112) and of odd
// ones [368,416), input rows hi [112,152) and lo [152,192), dH hi [192,256) and
// lo [256,320); dW0 accumulates in [320,368), dW1 (one output) per point of the tile
// in [416,480).
constexpr uint32_t kColH = 0, kColDin0 = 64, kColDin1 = 368, kColInHi = 112, kColInLo = 112 + kK1, kColDhHi = 192, kColDhLo = 256,
                   kColDw0 = 320, kColDw1 = 416;

// K steps of D (+)= A[TMEM columns from a] B[shared memory, descriptor b]^T.
__device__ __forceinline__ void mma_chain(uint32_t d, uint32_t a, uint64_t b, int ksteps, uint32_t idesc,
                                          bool fresh) {
  for (int ks = 0; ks < ksteps; ++ks)
    tc::mma_ts(d, a + 8u * ks, b + 16u * ks, idesc, (fresh && ks == 0) ? 0u : 1u);
}

// With M members per quadrant group, member g handles levels g, g+M, g+2M, ...
// (coarse and fine levels mixed, which balances the scatter's shuffle and
// atomic work); with eight members (the backward kernels) levels g and 15 - g,
// which measured 1.3 % faster than g and g + 8 in the backward (the members
// scattering levels 1-4, whose same-cell groups cost the most, then also hold
// the cheapest fine levels).  Member g's 32/M features sit in permuted input
// columns (32/M)g .. (32/M)g + 32/M - 1.
// Warp index, known to the compiler to be the same on every lane: the level of
// a member then sits in uniform registers, its constants come by uniform loads
// and its branches need no reconvergence (a fifth of the forward's instructions).
__device__ __forceinline__ int uniform_warp() { return __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0); }

template <int M>
__device__ __forceinline__ int level_of(int g, int i) {
  if constexpr (M == 8) return i == 0 ? g : 15 - g;
  return g + M * i;
}

// Permuted input column -> column of W0 (or -1 for a zero column).
template <int M>
__device__ __forceinline__ int w0_col(int c, int L) {
  constexpr int kFpm = kXCol / M;  // features per member
  if (c < kXCol) {
    const int l = level_of<M>(c / kFpm, (c % kFpm) >> 1);
    return l < L ? 3 + 2 * l + (c & 1) : -1;
  }
  if (c < kXCol + 3) return c - kXCol;
  return -1;
}

// Table-gradient contributions of the warp's 32 points at one level; `value(f,
// d, x1, yz)` is the contribution of a point with cell fractions f and values d
// to the corner on side x1 of x and the sides of yz's bits 0 and 1 of y and z.
//  * Lanes sharing a cell are summed first: the cell of the first remaining
//    lane is matched exactly (three coordinates), and if it holds at least
//    kMinGroupLanes lanes their float2 contributions to the 8 corners are
//    summed by a reduce-scatter over the warp (corner bit 2 follows lane bit
//    4, bit 1 lane bit 3, bit 0 lane bit 2) and added by one float2 atomic per
//    corner, issued together by lanes 0, 4, ..., 28; up to kMaxCellGroups cells.
//  * The points left are added by lane pairs, as gather_corners reads them: two
//    lanes add one point's two x corners together, which lie in one line 15
//    times of 16, so the pair is one request to the L2 (4.25 a point and level,
//    against 6 with a lane adding all its corners, aligned pairs as one 16-byte
//    atomic) and no lane takes a path of its own.
// Measured on the bench workload's backward (two rounds each): groups of
// >= 8 lanes, at most 2 per level, beat >= 4 lanes / 4 groups by 2 %, and
// smaller groups or more of them were slower (their shuffles cost more than
// the L2 requests they save).
constexpr int kMaxCellGroups = 2;
constexpr int kMinGroupLanes = 8;

template <int ND, typename Value>
__device__ __forceinline__ void scatter_level(const GridDev& gd, int l, const PointPair& q, const float d[ND],
                                              bool live, float2* gt2, int lane, const Value& value) {
  constexpr unsigned kAll = 0xffffffffu;
  const LevelDev lv = gd.lv[l];
  float2* t = gt2 + lv.offset;
  float fa[3], fb[3];
  uint32_t ca[3], cb[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float pa = __fmaf_rn(lv.scale, q.a[k], 0.5f), pb = __fmaf_rn(lv.scale, q.b[k], 0.5f);
    fa[k] = __fsub_rn(pa, floorf(pa));
    fb[k] = __fsub_rn(pb, floorf(pb));
    ca[k] = (uint32_t)__float2int_rd(pa);
    cb[k] = (uint32_t)__float2int_rd(pb);
  }
  const uint32_t cell[3] = {q.odd ? cb[0] : ca[0], q.odd ? cb[1] : ca[1], q.odd ? cb[2] : ca[2]};
  unsigned rest = __ballot_sync(kAll, live);
  for (int it = 0; it < kMaxCellGroups && rest != 0u; ++it) {
    const int ld = __ffs(rest) - 1;
    const uint32_t c0 = __shfl_sync(kAll, cell[0], ld);
    const uint32_t c1 = __shfl_sync(kAll, cell[1], ld);
    const uint32_t c2 = __shfl_sync(kAll, cell[2], ld);
    const bool in = ((rest >> lane) & 1u) & (cell[0] == c0) & (cell[1] == c1) & (cell[2] == c2);
    const unsigned gm = __ballot_sync(kAll, in);
    if (__popc(gm) < kMinGroupLanes) break;  // the same decision on every lane
    const float f[3] = {q.odd ? fb[0] : fa[0], q.odd ? fb[1] : fa[1], q.odd ? fb[2] : fa[2]};
    float v[16];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float2 c = value(f, d, (k & 1) != 0, k >> 1);
      v[2 * k] = in ? c.x : 0.0f;
      v[2 * k + 1] = in ? c.y : 0.0f;
    }
    float a8[8], a4[4], a2[2];
    bool up = lane & 16;
#pragma unroll
    for (int i = 0; i < 8; ++i) a8[i] = (up ? v[i + 8] : v[i]) + __shfl_xor_sync(kAll, up ? v[i] : v[i + 8], 16);
    up = lane & 8;
#pragma unroll
    for (int i = 0; i < 4; ++i) a4[i] = (up ? a8[i + 4] : a8[i]) + __shfl_xor_sync(kAll, up ? a8[i] : a8[i + 4], 8);
    up = lane & 4;
#pragma unroll
    for (int i = 0; i < 2; ++i) a2[i] = (up ? a4[i + 2] : a4[i]) + __shfl_xor_sync(kAll, up ? a4[i] : a4[i + 2], 4);
#pragma unroll
    for (int sft = 2; sft > 0; sft >>= 1) {
      a2[0] += __shfl_xor_sync(kAll, a2[0], sft);
      a2[1] += __shfl_xor_sync(kAll, a2[1], sft);
    }
    const int k = lane >> 2;  // corner summed into lanes 4k..4k+3
    if ((lane & 3) == 0)
      atomicAdd(t + corner_at(lv, c0 + (k & 1), c1 + ((k >> 1) & 1), c2 + (k >> 2)), make_float2(a2[0], a2[1]));
    rest &= ~gm;
  }
  if (rest == 0u) return;
  float da[ND], db[ND];
#pragma unroll
  for (int i = 0; i < ND; ++i) {
    const float o = __shfl_xor_sync(kAll, d[i], 1);
    da[i] = q.odd ? o : d[i];
    db[i] = q.odd ? d[i] : o;
  }
  uint32_t idx[4];
  if ((rest >> (lane & ~1)) & 1u) {
    corner_quad(lv, ca[0] + q.odd, ca[1], ca[2], idx);
#pragma unroll
    for (int j = 0; j < 4; ++j) atomicAdd(t + idx[j], value(fa, da, q.odd != 0u, j));
  }
  if ((rest >> (lane | 1)) & 1u) {
    corner_quad(lv, cb[0] + (q.odd ^ 1u), cb[1], cb[2], idx);
#pragma unroll
    for (int j = 0; j < 4; ++j) atomicAdd(t + idx[j], value(fb, db, q.odd == 0u, j));
  }
}

// Trilinear weight of a corner.
__device__ __forceinline__ float corner_weight(const float f[3], bool x1, int yz) {
  const float wx = x1 ? f[0] : __fsub_rn(1.0f, f[0]);
  const float wy = (yz & 1) ? f[1] : __fsub_rn(1.0f, f[1]);
  const float wz = (yz & 2) ? f[2] : __fsub_rn(1.0f, f[2]);
  return __fmul_rn(__fmul_rn(wx, wy), wz);
}

// W0 (64, din) -> B1 (N = 64 hidden, K = 40 inputs, K-major) hi/lo, and, with
// W0T, W0^T -> B2 (N = 48 inputs, K = 64 hidden, K-major) hi/lo.  A thread takes four
// columns of a row, which lie together in a core matrix (one 16-byte store each
// for hi and lo), a warp eight rows by four such groups: no two lanes of a store
// in a bank, 8 to 16 lines a load.  Every CTA stages, so a small launch's time is
// to a good part this: element by element a 2,053-point forward took 13.3 us, now 9.9,
// and a backward 19.0 us, now 16.0 (with 32-bit tile counts).
template <int M, bool W0T>
__device__ __forceinline__ void stage_w0(const FieldArgs& a, uint8_t* b1_hi, uint8_t* b1_lo, uint8_t* b2_hi,
                                         uint8_t* b2_lo) {
  constexpr int kGroups = (W0T ? kN2 : kK1) / 4;
  for (int e = threadIdx.x; e < kH * kGroups; e += blockDim.x) {
    const int item = e >> 3, block = item / kGroups, cg = item - block * kGroups, j = 8 * block + (e & 7);
    float v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int src = 4 * cg + k < kK1 ? w0_col<M>(4 * cg + k, a.g.L) : -1;
      v[k] = src >= 0 ? a.w0[j * a.din + src] : 0.0f;
    }
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) tc::tf32_split(v[k], hi[k], lo[k]);
    if (4 * cg < kK1) {
      const uint32_t o1 = tc::kmajor_offset(j, 4 * cg, kK1);
      *reinterpret_cast<uint4*>(b1_hi + o1) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      *reinterpret_cast<uint4*>(b1_lo + o1) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
    if constexpr (W0T) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t o2 = tc::kmajor_offset(4 * cg + k, j, kH);
        *reinterpret_cast<uint32_t*>(b2_hi + o2) = hi[k];
        *reinterpret_cast<uint32_t*>(b2_lo + o2) = lo[k];
      }
    }
  }
}

// BF16 first-layer operands: K padded to 48, core matrices of 8 rows x 8
// elements (16 bytes), K-adjacent core matrices contiguous (LBO 128 bytes),
// 8-row groups kBf16Sbo bytes apart.
constexpr int kK1b = 48;
constexpr uint32_t kBf16Sbo = (kK1b / 8) * 128u;

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);  // .x (lower K) in the low half
  return *reinterpret_cast<const uint32_t*>(&v);
}

// W0 (64, din) -> B (N = 64 hidden, K = 48 permuted inputs, K-major), BF16.
template <int M>
__device__ void stage_w0_bf16(const FieldArgs& a, uint8_t* b) {
  for (int e = threadIdx.x; e < kH * kK1b; e += blockDim.x) {
    const int j = e / kK1b, c = e - j * kK1b;
    const int src = c < kK1 ? w0_col<M>(c, a.g.L) : -1;
    const float v = src >= 0 ? a.w0[j * a.din + src] : 0.0f;
    const uint32_t off = (uint32_t)(j >> 3) * kBf16Sbo + (uint32_t)(c >> 3) * 128u + (uint32_t)(j & 7) * 16u +
                         (uint32_t)(c & 7) * 2u;
    *reinterpret_cast<__nv_bfloat16*>(b + off) = __float2bfloat16_rn(v);
  }
}

__device__ __forceinline__ void load_point(const FieldArgs& a, int64_t p, int64_t n, float x[3]) {
  if (p < n) {
    x[0] = a.x[3 * p];
    x[1] = a.x[3 * p + 1];
    x[2] = a.x[3 * p + 2];
  } else {
    x[0] = x[1] = x[2] = 0.0f;
  }
}
__device__ __forceinline__ void load_point(const float* __restrict__ p, bool live, float x[3]) {
#pragma unroll
  for (int d = 0; d < 3; ++d) x[d] = live ? p[d] : 0.0f;
}
// The tiles of one CTA of a persistent grid: blockIdx.x, blockIdx.x + gridDim.x,
// ...; every one but the last of all tiles is whole.  Step counters are 32-bit
// and the same on every lane, so a step's bookkeeping is a few instructions.
struct TileWalk {
  int count;        // this CTA's tiles
  int whole;        // of which whole (the others: one of `rest` points, or none)
  int rest;
  int64_t first;    // first point of the CTA's first tile
  int64_t stride;   // points between its tiles
  __device__ __forceinline__ explicit TileWalk(int64_t n) {
    // (tiles fit 32 bits: 2^32 of them would be 6 TB of coordinates)
    const uint32_t tiles = (uint32_t)((n + kTile - 1) / kTile), full = (uint32_t)(n / kTile);
    const uint32_t b = blockIdx.x, s = gridDim.x;
    count = b < tiles ? (int)((tiles - b + s - 1) / s) : 0;
    whole = b < full ? (int)((full - b + s - 1) / s) : 0;
    rest = (int)(n - (int64_t)full * kTile);
    first = (int64_t)b * kTile;
    stride = (int64_t)s * kTile;
  }
  // point pt of the CTA's i-th tile is below n
  __device__ __forceinline__ bool live(int i, int pt) const { return i < whole || (i < count && pt < rest); }
};

// Output gradients at go (zeros for a point that is not live).
template <int OC>
__device__ __forceinline__ void load_grad(const float* __restrict__ p, int cols, bool live, float go[OC]) {
#pragma unroll
  for (int o = 0; o < OC; ++o) go[o] = (live && o < cols) ? p[o] : 0.0f;
}

// Member g's levels of a point from the encoding cache, whose level l is at
// enc[l * cap] (zeros for a point that is not live and past the active levels, as
// encode_group gives).  Read once, so streamed past L2.
template <int M>
__device__ __forceinline__ void load_enc(const float2* enc, int64_t cap, int g, int active, bool live,
                                         float e[2 * (16 / M)]) {
#pragma unroll
  for (int i = 0; i < 16 / M; ++i) {
    float2 v = make_float2(0.0f, 0.0f);
    if (live && level_of<M>(g, i) < active) v = __ldcs(enc + level_of<M>(g, i) * cap);
    e[2 * i] = v.x;
    e[2 * i + 1] = v.y;
  }
}

// Encoding of member g's levels of the lane's point: e[2i + f] for level
// level_of(g, i); zeros past the active levels and for points that are not live.
template <int M, bool FP32 = false>
__device__ __forceinline__ void encode_group(const FieldArgs& a, int g, bool live, const PointPair& q,
                                             float e[2 * (16 / M)]) {
  const bool any = __any_sync(0xffffffffu, live);
#pragma unroll
  for (int i = 0; i < 16 / M; ++i) {
    const int l = level_of<M>(g, i);
    float e0 = 0.0f, e1 = 0.0f;
    if (any && l < a.active) encode_level_pair<FP32>(a, l, q, e0, e1);
    e[2 * i] = live ? e0 : 0.0f;
    e[2 * i + 1] = live ? e1 : 0.0f;
  }
}

// Sums 8 per-lane values over the warp by a reduce-scatter (9 shuffles):
// lanes 4m .. 4m+3 end with the sum of value m.
__device__ __forceinline__ float warp_reduce_scatter8(const float v[8], int lane) {
  constexpr unsigned kAll = 0xffffffffu;
  float a4[4], a2[2];
  bool up = lane & 16;
#pragma unroll
  for (int i = 0; i < 4; ++i) a4[i] = (up ? v[i + 4] : v[i]) + __shfl_xor_sync(kAll, up ? v[i] : v[i + 4], 16);
  up = lane & 8;
#pragma unroll
  for (int i = 0; i < 2; ++i) a2[i] = (up ? a4[i + 2] : a4[i]) + __shfl_xor_sync(kAll, up ? a4[i] : a4[i + 2], 8);
  up = lane & 4;
  float a1 = (up ? a2[1] : a2[0]) + __shfl_xor_sync(kAll, up ? a2[0] : a2[1], 4);
  a1 += __shfl_xor_sync(kAll, a1, 2);
  a1 += __shfl_xor_sync(kAll, a1, 1);
  return a1;
}

template <bool EVEN>
__device__ __forceinline__ void tf32_split(float x, uint32_t& hi, uint32_t& lo) {
  if constexpr (EVEN) tc::tf32_split_even(x, hi, lo);
  else tc::tf32_split(x, hi, lo);
}
template <bool EVEN = false>
__device__ __forceinline__ void st_split8(uint32_t ta_hi, uint32_t ta_lo, const float v[8]) {
  uint32_t hi[8], lo[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) tf32_split<EVEN>(v[i], hi[i], lo[i]);
  tc::tmem_st8(ta_hi, hi);
  tc::tmem_st8(ta_lo, lo);
}
template <bool EVEN = false>
__device__ __forceinline__ void st_split4(uint32_t ta_hi, uint32_t ta_lo, const float v[4]) {
  uint32_t hi[4], lo[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) tf32_split<EVEN>(v[i], hi[i], lo[i]);
  tc::tmem_st4(ta_hi, hi);
  tc::tmem_st4(ta_lo, lo);
}
// Stores N (4, 8 or 16) values, split into TF32 hi/lo, at columns c_hi / c_lo.
template <int N, bool EVEN = false>
__device__ __forceinline__ void st_split(uint32_t ta_hi, uint32_t ta_lo, const float* v) {
  if (N == 4) {
    st_split4<EVEN>(ta_hi, ta_lo, v);
  } else {
#pragma unroll
    for (int i = 0; i < N; i += 8) st_split8<EVEN>(ta_hi + i, ta_lo + i, v + i);
  }
}

// ---------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------
// M members per TMEM lane quadrant: 128 M threads; member g owns levels
// level_of<M>(g, i), input columns (32/M)g .. and hidden units (64/M)g ...
// M = 4: 512 threads, two CTAs per SM; M = 8: 1024 threads, one CTA per SM.
constexpr int kFwdMembers = 4;

template <int M>
struct FwdSmem {
  static constexpr uint32_t b1_hi = 0, b1_lo = 10240, w1 = 20480, b0 = 24576, b1 = 24832,
                            bar = 24896, slot = bar + 8, part = slot + 8;
  // partial outputs, one buffer for each of two tiles in flight
  template <bool ONE>
  static constexpr uint32_t part_bytes = M * kTile * (ONE ? 1 : kDoutMax) * 4;
  // more than 228/3 KB, so at most two CTAs (2 x 256 TMEM columns) per SM
  template <bool ONE>
  static constexpr size_t bytes = ONE ? 80 * 1024 : 96 * 1024;
};
static_assert(FwdSmem<4>::part + 2 * FwdSmem<4>::part_bytes<false> <= FwdSmem<4>::bytes<false>,
              "forward shared memory map");

// N (a multiple of 4) consecutive floats of shared memory at a 16-byte boundary.
template <int N>
__device__ __forceinline__ void lds_n(const float* p, float* v) {
#pragma unroll
  for (int i = 0; i < N; i += 4) {
    const float4 q = *reinterpret_cast<const float4*>(p + i);
    v[i] = q.x;
    v[i + 1] = q.y;
    v[i + 2] = q.z;
    v[i + 3] = q.w;
  }
}

template <int N>
__device__ __forceinline__ void tmem_ld_n(uint32_t ta, float* v) {
  if constexpr (N == 16) tc::tmem_ld16(ta, v);
  else if constexpr (N == 8) tc::tmem_ld8(ta, v);
  else tc::tmem_ld4(ta, v);
}

// Segments of one forward launch: point sets that each have their own table,
// level geometry and MLP (several objects' queries in one persistent launch).
constexpr int kMaxSegments = 4;
struct FieldSegments {
  int n;
  FieldArgs seg[kMaxSegments];
};

// ONE: a single output column (the sdf; every training call), else up to kDoutMax.
// Each CTA works through the segments in order: it stages segment s's
// weights, processes its share of s's tiles (persistent, strided by the
// grid), then moves on; one launch of one segment is the ordinary forward.
//
// The tiles are pipelined so that a tile costs one block barrier: a step gathers
// tile i + 1's encoding while tile i's MMAs run, then (they have long finished)
// stores it as the next A operand, reads tile i's hidden layer, and after
// the barrier issues tile i + 1's MMAs and sums tile i's outputs over the members.
// With the phases of one tile after another (encode, MMA wait, hidden layer, sum:
// four barriers) a warp spent a quarter of its stalls at them.  With the uniform
// level indices, the 256^3 SDF lattice went from 5.02 to 4.44 ms and 500 k training
// points from 132 to 102 us (with the paired gathers); with x fastest on the lattice
// and the precision and staging below, 3.0 ms (5.7 G points/s) and 94 us.  What bounds
// it now is instructions (4,175 per 32 points, issue slots 58 % taken) and the L1 data
// pipe (60 %).
// FP32: no segment asks for a lower precision (the FP16 table, one-pass products).
template <bool ONE, int M, bool FP32>
__global__ void __launch_bounds__(128 * M, M == 4 ? 2 : 1)
field_fwd_tc_kernel(const __grid_constant__ FieldSegments segs) {
  constexpr int kOc = ONE ? 1 : kDoutMax;
  constexpr int kNt = 128 * M;      // threads
  constexpr int kLpm = 16 / M;      // levels per member
  constexpr int kFpm = 2 * kLpm;    // input features per member
  constexpr int kHpm = kH / M;      // hidden units per member
  using Sm = FwdSmem<M>;
  extern __shared__ __align__(1024) uint8_t sm[];
  float* s_w1 = reinterpret_cast<float*>(sm + Sm::w1);
  float* s_b0 = reinterpret_cast<float*>(sm + Sm::b0);
  float* s_b1 = reinterpret_cast<float*>(sm + Sm::b1);
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + Sm::bar);
  uint32_t* slot = reinterpret_cast<uint32_t*>(sm + Sm::slot);
  const int t = threadIdx.x, warp = uniform_warp(), lane = t & 31;
  const int q = warp & 3, g = warp >> 2;
  const int pt = 32 * q + lane;  // point within the tile == TMEM lane

  // after the wait: a CTA that holds tensor memory never waits for another grid
  chain_wait();
  if (warp == 0) {
    tc::tmem_alloc(slot, kCols);
    tc::tmem_relinquish();
  }
  if (t == 0) tc::mbar_init(bar, 2);  // one commit each from threads 0 and 32
  const uint32_t lb = (uint32_t)(32 * q);
  const uint32_t s_b1_hi = tc::smem_u32(sm + Sm::b1_hi), s_b1_lo = tc::smem_u32(sm + Sm::b1_lo);
  uint32_t phase = 0;
  int buf = 0;
  bool ok = true;
  uint32_t tbase = 0;

  for (int si = 0; si < segs.n && ok; ++si) {
    const FieldArgs& a = segs.seg[si];
    const bool bf16 = !FP32 && a.bf16, one_pass = !FP32 && a.one_pass;
    const int oc = a.out_cols;
    const float inv_beta = 1.0f / a.beta;
    if (si > 0) __syncthreads();     // the previous segment's last tile is done with the weights
    if (bf16) {
      if constexpr (M == 4) stage_w0_bf16<M>(a, sm + Sm::b1_hi);
    } else {
      stage_w0<M, false>(a, sm + Sm::b1_hi, sm + Sm::b1_lo, nullptr, nullptr);
    }
    for (int e = t; e < oc * kH; e += kNt) s_w1[e] = a.w1[e];
    if (t < kH) s_b0[t] = a.b0[t];
    if (t < kDoutMax) s_b1[t] = t < oc ? a.b1[t] : 0.0f;
    tc::fence_proxy_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    tbase = *slot;
    chain_release();   // with its tensor memory allocated: a successor's CTA may want the rest

    const TileWalk walk(effective_n(a));
    // this point's coordinates one tile ahead: the stream read overlaps a tile
    float xn[3] = {0.0f, 0.0f, 0.0f};
    const float* x_ptr = a.x + 3 * (walk.first + pt);
    load_point(x_ptr, walk.live(0, pt), xn);
    int64_t p = walk.first + pt;   // the point to encode; its predecessor's output is written
    for (int i = 0; i <= walk.count && walk.count > 0; ++i) {
      const bool more = i < walk.count, pending = i > 0;
      const bool live = more && walk.live(i, pt);
      const float x[3] = {xn[0], xn[1], xn[2]};
      float e[kFpm];
      if (more) {
        x_ptr += 3 * walk.stride;
        load_point(x_ptr, walk.live(i + 1, pt), xn);
        encode_group<M, FP32>(a, g, live, make_pair(x, lane), e);
        if (a.enc_out && live) {
#pragma unroll
          for (int k = 0; k < kLpm; ++k) {
            const int l = level_of<M>(g, k);
            if (l < a.active) __stcs(a.enc_out + (int64_t)l * a.cap + p, make_float2(e[2 * k], e[2 * k + 1]));
          }
        }
      }
      bool got = true;
      if (pending) {
        got = __all_sync(0xffffffffu, tc::mbar_wait_bounded(bar, phase));
        phase ^= 1u;
        tc::fence_after_sync();
      }
      if (more && got) {  // the MMAs that read the previous rows are done
        if (bf16) {
          // BF16 pairs: member g's 8 features in columns 4g .. 4g + 3, x (and
          // the zero padding up to K = 48) in columns 16 .. 23
          if constexpr (M == 4) {
            uint32_t pk[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) pk[i] = pack_bf16(e[2 * i], e[2 * i + 1]);
            tc::tmem_st4(tc::taddr(tbase, lb, kFwdColInHi + 4 * g), pk);
            if (g == 0) {
              const uint32_t xp[8] = {pack_bf16(x[0], x[1]), pack_bf16(x[2], 0.0f), 0u, 0u, 0u, 0u, 0u, 0u};
              tc::tmem_st8(tc::taddr(tbase, lb, kFwdColInHi + kXCol / 2), xp);
            }
          }
        } else {
          st_split<kFpm>(tc::taddr(tbase, lb, kFwdColInHi + kFpm * g), tc::taddr(tbase, lb, kFwdColInLo + kFpm * g), e);
          if (g == 0) {
            const float xv[8] = {x[0], x[1], x[2], 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
            st_split8(tc::taddr(tbase, lb, kFwdColInHi + kXCol), tc::taddr(tbase, lb, kFwdColInLo + kXCol), xv);
          }
        }
      }
      // hidden units kHpm g .. kHpm g + kHpm - 1 of the previous point -> partial
      // outputs; one output: a column of 128 floats per member (no two lanes in a bank)
      constexpr int kPs = ONE ? 1 : kDoutMax;
      float* s_part = reinterpret_cast<float*>(sm + Sm::part) + buf * (M * kTile * kPs);
      if (pending && got) {
        float h[kHpm];
        tmem_ld_n<kHpm>(tc::taddr(tbase, lb, kFwdColH0 + kHpm * g), h);
        if (!one_pass && !bf16) {
          float h1[kHpm];
          tmem_ld_n<kHpm>(tc::taddr(tbase, lb, kFwdColH1 + kHpm * g), h1);
          tc::tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < kHpm; ++i) h[i] += h1[i];
        }
        tc::tmem_wait_ld();
        float part[kOc];
#pragma unroll
        for (int o = 0; o < kOc; ++o) part[o] = 0.0f;
        float b0v[kHpm];
        lds_n<kHpm>(s_b0 + kHpm * g, b0v);
        if constexpr (ONE) {
          float w1v[kHpm];
          lds_n<kHpm>(s_w1 + kHpm * g, w1v);
#pragma unroll
          for (int i = 0; i < kHpm; ++i) {
            const float act = softplus_fast(h[i] + b0v[i], a.beta, inv_beta, a.thresh);
            part[0] = fmaf(w1v[i], act, part[0]);
          }
        } else {
#pragma unroll
          for (int i = 0; i < kHpm; ++i) {
            const int j = kHpm * g + i;
            const float act = softplus_fast(h[i] + b0v[i], a.beta, inv_beta, a.thresh);
#pragma unroll
            for (int o = 0; o < kOc; ++o)
              if (o < oc) part[o] = fmaf(s_w1[o * kH + j], act, part[o]);
          }
        }
#pragma unroll
        for (int o = 0; o < kOc; ++o)
          if (o < oc) s_part[(g * kTile + pt) * kPs + o] = part[o];
      }
      tc::tmem_wait_st();
      tc::fence_before_sync();
      if (!__syncthreads_and(got)) {
        ok = false;
        break;
      }
      if (more && (t == 0 || t == 32)) {  // H = IN W0^T, M=128, N=64, K=40 (BF16: K=48, three K=16 steps)
        tc::fence_after_sync();
        if (bf16) {
          if (t == 0) {
            const uint64_t wb = tc::smem_desc(s_b1_hi, 128u, kBf16Sbo);
            for (int ks = 0; ks < kK1b / 16; ++ks)
              tc::mma_ts_f16(tc::taddr(tbase, 0, kFwdColH0), tc::taddr(tbase, 0, kFwdColInHi + 8u * ks),
                             wb + (uint64_t)((256u * ks) >> 4), tc::idesc_bf16(kTile, kH), ks > 0 ? 1u : 0u);
          }
        } else {
          const uint32_t idesc = tc::idesc_tf32(kTile, kH);
          const uint32_t sbo = (kK1 / 4) * 128u;
          const uint64_t w_hi = tc::smem_desc(s_b1_hi, 128u, sbo), w_lo = tc::smem_desc(s_b1_lo, 128u, sbo);
          if (t == 0) {
            mma_chain(tc::taddr(tbase, 0, kFwdColH0), tc::taddr(tbase, 0, kFwdColInHi), w_hi, kK1 / 8, idesc, true);
          } else if (!one_pass) {
            mma_chain(tc::taddr(tbase, 0, kFwdColH1), tc::taddr(tbase, 0, kFwdColInLo), w_hi, kK1 / 8, idesc, true);
            mma_chain(tc::taddr(tbase, 0, kFwdColH1), tc::taddr(tbase, 0, kFwdColInHi), w_lo, kK1 / 8, idesc, false);
          }
        }
        tc::mma_commit(bar);
      }
      if (pending && g == 0 && walk.live(i - 1, pt)) {
        float* out = a.out + (p - walk.stride) * oc;
        for (int o = 0; o < oc; ++o) {
          float sum = s_b1[o];
#pragma unroll
          for (int m = 0; m < M; ++m) sum += s_part[(m * kTile + pt) * kPs + o];
          out[o] = sum;
        }
      }
      p += walk.stride;
      buf ^= 1;
    }
  }
  if (!ok) {
    if (t == 0) {
      for (int si = 0; si < segs.n; ++si)
        if (segs.seg[si].status) atomicOr(segs.seg[si].status, SN_STATUS_TIMEOUT);
    }
    (void)tc::mbar_wait_bounded(bar, phase ^ 1u);
  }
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(*slot, kCols);
}

// ---------------------------------------------------------------------------
// backward
// ---------------------------------------------------------------------------
struct BwdSmem {
  static constexpr uint32_t b1_hi = 0, b1_lo = 10240, b2_hi = 20480, b2_lo = 32768, a3 = 45056,
                            b3_hi = a3 + 16 * kSboP, b3_lo = b3_hi + 6 * kSboP, w1 = b3_lo + 6 * kSboP,
                            b0 = w1 + kDoutMax * kH * 4, dx = b0 + kH * 4, bar = dx + 8 * kTile * 3 * 4,
                            slot = bar + 8, dw1 = slot + 8, end = dw1 + kDoutMax * kH * 4;
};
constexpr size_t kBwdSmemBytes = BwdSmem::end;
static_assert(BwdSmem::end <= 227 * 1024, "backward shared memory map");

__device__ __forceinline__ void st_smem_u32(uint8_t* base, uint32_t off, uint32_t v) {
  *reinterpret_cast<uint32_t*>(base + off) = v;
}

// 3xTF32 D = A W^T with A in TMEM (hi at a_hi, lo at a_lo), W staged hi/lo; the
// hi.hi product alone where one pass is asked for.  The tensor core truncates as it
// accumulates, so the small products go first: added onto the hi.hi sums they left
// dL/dx 7e-7 off (relative norm against 64 bits, 65,536 points), this way 2.5e-7,
// what three separate sums leave; the other gradients are no further off than with
// those either (500,003 points, three seeds: table 2.2-3.1e-7, weight_v of the first
// layer 1.0-1.7e-5, its bias 1.6-4.9e-6, both ways).
__device__ __forceinline__ void mma_3x(uint32_t d, uint32_t a_hi, uint32_t a_lo, uint64_t w_hi, uint64_t w_lo,
                                       int ksteps, uint32_t idesc, bool one_pass = false) {
  if (!one_pass) {
    mma_chain(d, a_lo, w_hi, ksteps, idesc, true);
    mma_chain(d, a_hi, w_lo, ksteps, idesc, false);
  }
  mma_chain(d, a_hi, w_hi, ksteps, idesc, one_pass);
}

// Third MMA: dW0 += [dH_hi; dH_lo]^T-rows x IN^T (M=128, N=48, K=128 points),
// accumulated in TMEM over all of the CTA's tiles.
__device__ __forceinline__ void issue_mma3(uint32_t tbase, const uint8_t* sm, bool first_tile, bool one_pass) {
  const uint32_t s_a3 = tc::smem_u32(sm + BwdSmem::a3);
  const uint32_t s_b3_hi = tc::smem_u32(sm + BwdSmem::b3_hi), s_b3_lo = tc::smem_u32(sm + BwdSmem::b3_lo);
  const uint32_t idesc = tc::idesc_tf32(kTile, kN2);
  const uint32_t d3 = tc::taddr(tbase, 0, kColDw0);
  const uint64_t da = tc::smem_desc(s_a3, kLboP, kSboP), dbh = tc::smem_desc(s_b3_hi, kLboP, kSboP),
                 dbl = tc::smem_desc(s_b3_lo, kLboP, kSboP);
  for (int ks = 0; ks < kTile / 8; ++ks) {
    const uint64_t k0 = (2u * kLboP * ks) >> 4;
    tc::mma_ss(d3, da + k0, dbh + k0, idesc, (first_tile && ks == 0) ? 0u : 1u);
    if (!one_pass) tc::mma_ss(d3, da + k0, dbl + k0, idesc, 1);
  }
}

// Adds the CTA's dW0 and db0 (TMEM columns from ta: lanes 0..63 hold the products
// of the hi rows, 64..127 those of the lo rows) to the gradients; every thread
// of the CTA takes part.  Both halves are summed in shared memory (`sums`: 64 x
// din weights, then 64 biases) and added in the weights' own order: 71 requests a
// CTA.  Added by the lanes that hold them, two to an address and 140 bytes apart,
// they were 4,600 requests a CTA to the same 70 lines, ~50 us of every launch.
template <int M>
__device__ __forceinline__ void flush_dw0(const FieldArgs& a, uint32_t ta, float* sums) {
  const int t = threadIdx.x, warp = uniform_warp(), pt = 32 * (warp & 3) + (t & 31), j = pt & (kH - 1);
  const int nw = kH * a.din;
  for (int half = 0; half < 2; ++half) {
    if (warp < 4 && (warp >> 1) == half) {
#pragma unroll
      for (int c0 = 0; c0 < kN2; c0 += 16) {
        float v[16];
        tc::tmem_ld16(ta + c0, v);
        tc::tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const int c = c0 + i, col = c < kK1 ? w0_col<M>(c, a.g.L) : -1;
          float* s = c == kOnesRow ? sums + nw + j : col >= 0 ? sums + j * a.din + col : nullptr;
          if (s) *s = half ? *s + v[i] : v[i];
        }
      }
    }
    __syncthreads();
  }
  if (a.grad_w0)
    for (int e = t; e < nw; e += blockDim.x)
      if (sums[e] != 0.0f) atomicAdd(a.grad_w0 + e, sums[e]);
  if (a.grad_b0 && t < kH) atomicAdd(a.grad_b0 + t, sums[nw + t]);
}

// A block's part of element e of the output layer's weight gradient.  In double
// where the caller has room for the sums: 152 parts of 500,003 points cancel, and added
// in float as they arrive they left the one gradient of weight_g that is not zero up to
// 1.5e-6 off, another amount at every call.
__device__ __forceinline__ void add_dw1(const FieldArgs& a, int e, double s) {
  if (s == 0.0) return;
  if (a.w1_sums)
    atomicAdd(a.w1_sums + e, s);
  else if (a.grad_w1)
    atomicAdd(a.grad_w1 + e, (float)s);
}

// M members per TMEM lane quadrant: 128 M threads, each member owning 16/M
// levels, 32/M input columns and 64/M hidden units of its 32 points.
//
// The tiles are pipelined over three stages, so a tile costs one block barrier
// and no MMA is waited for right after it is issued.  Step i
//   turns H of tile i into dH (TMEM, and dH^T in shared memory), copies tile i's
//   input rows to IN^T, and stores tile i + 1's input rows;
//   barrier; issues the MMAs dIN(i), H(i + 1) and dW0 += dH(i)^T IN(i);
//   scatters tile i - 1 while they run.
// A tile at a time (three barriers, two MMA round trips) the barriers were the
// largest stall: every phase waited for its slowest warp.  What bounds it now is
// instructions (issue slots 56 % taken, some 8,500 a warp's 32 points) and that
// barrier; the encoding cache and dL/dx are template arguments because their
// branches and registers showed: 500,003 cached points took 204 us, 195 with dW1
// summed per lane and TF32 rounded to even, 189 with the two as arguments, 198 with
// the softplus derivative's subnormals.  (The warps of a
// quadrant taking levels one by one from a shared counter, instead of owning two
// each, evened their arrival but gave nothing: 0.962 against 0.943 ms an
// iteration.)
constexpr int kBwdMembers = 8;

// DX: dL/dx may be wanted.  FP32: an FP32 table and three-pass products (one-pass
// products keep the rounding of the forward's operands, ties away: a tie is a whole
// TF32 step there).
template <bool ONE, int M, bool CACHED, bool DX, bool FP32>
__global__ void __launch_bounds__(128 * M, 1) field_bwd_tc_kernel(const __grid_constant__ FieldArgs a) {
  constexpr int kOc = ONE ? 1 : kDoutMax;
  constexpr int kNt = 128 * M;      // threads
  constexpr int kLpm = 16 / M;      // levels per member
  constexpr int kFpm = 2 * kLpm;    // input features per member
  constexpr int kHpm = kH / M;      // hidden units per member
  static_assert(kHpm == 8 && kFpm == 4, "eight members per quadrant");
  extern __shared__ __align__(1024) uint8_t sm[];
  float* s_w1 = reinterpret_cast<float*>(sm + BwdSmem::w1);
  float* s_b0 = reinterpret_cast<float*>(sm + BwdSmem::b0);
  float* s_dx = reinterpret_cast<float*>(sm + BwdSmem::dx);
  uint8_t* a3 = sm + BwdSmem::a3;
  uint8_t* b3_hi = sm + BwdSmem::b3_hi;
  uint8_t* b3_lo = sm + BwdSmem::b3_lo;
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + BwdSmem::bar);  // a step's three MMA groups
  uint32_t* slot = reinterpret_cast<uint32_t*>(sm + BwdSmem::slot);
  const int t = threadIdx.x, warp = uniform_warp(), lane = t & 31;
  const int q = warp & 3, g = warp >> 2;
  const int pt = 32 * q + lane;
  const int oc = a.out_cols;
  const float inv_beta = 1.0f / a.beta;
  const bool want_table = a.grad_table != nullptr;
  const bool one_pass = !FP32 && a.one_pass;
  const bool want_x = DX && a.grad_x != nullptr;

  chain_wait();   // before the tensor memory, as in the forward
  stage_w0<M, true>(a, sm + BwdSmem::b1_hi, sm + BwdSmem::b1_lo, sm + BwdSmem::b2_hi, sm + BwdSmem::b2_lo);
  for (int e = t; e < oc * kH; e += kNt) s_w1[e] = a.w1[e];
  if (t < kH) s_b0[t] = a.b0[t];
  float* s_dw1 = reinterpret_cast<float*>(sm + BwdSmem::dw1);
  for (int e = t; e < oc * kH; e += kNt) s_dw1[e] = 0.0f;
  // constant rows of IN^T: ones (hi) at kOnesRow, zeros above it
  for (int e = t; e < (kN2 - kOnesRow) * kTile; e += kNt) {
    const int r = kOnesRow + e / kTile, c = e % kTile;
    const uint32_t off = tc::kmajor_offset_strided(r, c, kLboP, kSboP);
    st_smem_u32(b3_hi, off, r == kOnesRow ? __float_as_uint(1.0f) : 0u);
    st_smem_u32(b3_lo, off, 0u);
  }
  if (warp == 0) {
    tc::tmem_alloc(slot, kBwdCols);
    tc::tmem_relinquish();
  }
  if (t == 0) tc::mbar_init(bar, 3);   // one commit from each of the three issuing threads
  tc::fence_proxy_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = *slot;
  chain_release();
  const uint32_t lb = (uint32_t)(32 * q);
  uint32_t phase = 0;
  int par = 0;   // step parity
  bool ok = true;

  const TileWalk walk(effective_n(a));
  // the tile whose input rows the next step stores: this point's coordinates
  // (unless the encoding cache holds what the member needs) and its member
  // levels, loaded one step ahead, as is the output gradient of the tile after
  // whose H is read
  const bool load_x = !CACHED || g == 0;
  float xn[3] = {0.0f, 0.0f, 0.0f}, gon[kOc], en[kFpm];
  const float* x_ptr = a.x + 3 * (walk.first + pt);             // of the tile that en and xn hold
  const float* go_ptr = a.grad_out + (walk.first + pt) * oc;
  const float2* enc_ptr = CACHED ? a.enc_in + walk.first + pt : nullptr;
  if (load_x) load_point(x_ptr, walk.live(0, pt), xn);
  if constexpr (CACHED) load_enc<M>(enc_ptr, a.cap, g, a.active, walk.live(0, pt), en);
  // i: the tile of the step's middle stage (H -> dH); the step before the first
  // tile fills the pipeline, the one after the last drains it
  for (int i = -1; i <= walk.count && walk.count > 0; ++i) {
    const bool has_in = i + 1 < walk.count, has_h = i >= 0 && i < walk.count, has_din = i > 0;
    const bool live_out = has_din && walk.live(i - 1, pt);
    float xo[3];  // the scattered point, read again (two tiles back, so in the L2)
    load_point(x_ptr - 6 * walk.stride, live_out, xo);
    float e[kFpm];
    if (has_in) {
      if constexpr (CACHED) {
#pragma unroll
        for (int k = 0; k < kFpm; ++k) e[k] = en[k];
      } else {
        encode_group<M, FP32>(a, g, walk.live(i + 1, pt), make_pair(xn, lane), e);
      }
    }
    bool got = true;
    if (i >= 0) {  // the MMAs of the previous step
      got = __all_sync(0xffffffffu, tc::mbar_wait_bounded(bar, phase));
      phase ^= 1u;
      tc::fence_after_sync();
    }
    if (has_h && got) {
      // ---- IN^T from the input rows (exact: the split values themselves) ----
      {
        float hi[kFpm], lo[kFpm];
        tc::tmem_ld4(tc::taddr(tbase, lb, kColInHi + kFpm * g), hi);
        tc::tmem_ld4(tc::taddr(tbase, lb, kColInLo + kFpm * g), lo);
        tc::tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < kFpm; ++i) {
          const uint32_t off = tc::kmajor_offset_strided(kFpm * g + i, pt, kLboP, kSboP);
          st_smem_u32(b3_hi, off, __float_as_uint(hi[i]));
          st_smem_u32(b3_lo, off, __float_as_uint(lo[i]));
        }
        if (g == 0) {
          tc::tmem_ld4(tc::taddr(tbase, lb, kColInHi + kXCol), hi);
          tc::tmem_ld4(tc::taddr(tbase, lb, kColInLo + kXCol), lo);
          tc::tmem_wait_ld();
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const uint32_t off = tc::kmajor_offset_strided(kXCol + i, pt, kLboP, kSboP);
            st_smem_u32(b3_hi, off, __float_as_uint(hi[i]));
            st_smem_u32(b3_lo, off, __float_as_uint(lo[i]));
          }
        }
      }
      // ---- dH for this member's hidden units kHpm g .. kHpm g + kHpm - 1 ----
      float go[kOc];
#pragma unroll
      for (int o = 0; o < kOc; ++o) go[o] = gon[o];
      float h[kHpm], b0v[kHpm];
      tc::tmem_ld8(tc::taddr(tbase, lb, kColH + kHpm * g), h);
      lds_n<kHpm>(s_b0 + kHpm * g, b0v);
      tc::tmem_wait_ld();
      float dh[kHpm], act[kHpm];
      if constexpr (ONE) {
        float w1v[kHpm];
        lds_n<kHpm>(s_w1 + kHpm * g, w1v);
#pragma unroll
        for (int i = 0; i < kHpm; ++i) {
          float sg;
          softplus_fwd_grad_fast(h[i] + b0v[i], a.beta, inv_beta, a.thresh, act[i], sg);
          dh[i] = go[0] * w1v[i] * sg;   // zero for a point that is not live: its go is
        }
      } else {
#pragma unroll
        for (int i = 0; i < kHpm; ++i) {
          const int j = kHpm * g + i;
          float sg;
          softplus_fwd_grad_fast(h[i] + b0v[i], a.beta, inv_beta, a.thresh, act[i], sg);
          float da = 0.0f;
#pragma unroll
          for (int o = 0; o < kOc; ++o)
            if (o < oc) da = fmaf(go[o], s_w1[o * kH + j], da);
          dh[i] = da * sg;
        }
      }
      st_split<kHpm, FP32>(tc::taddr(tbase, lb, kColDhHi + kHpm * g), tc::taddr(tbase, lb, kColDhLo + kHpm * g), dh);
#pragma unroll
      for (int i = 0; i < kHpm; ++i) {
        uint32_t hi, lo;
        tf32_split<FP32>(dh[i], hi, lo);
        st_smem_u32(a3, tc::kmajor_offset_strided(kHpm * g + i, pt, kLboP, kSboP), hi);
        st_smem_u32(a3, tc::kmajor_offset_strided(kH + kHpm * g + i, pt, kLboP, kSboP), lo);
      }
      // dW1[o][j] += sum over the points of g_o * act_j: one output, a sum per lane
      // (point of the tile) in TMEM, taken over the lanes after the last tile (a
      // warp's sum of eight values is 9 shuffles and some 35 instructions);
      // several outputs, summed over the warp here
      if constexpr (ONE) {
        const uint32_t ta = tc::taddr(tbase, lb, kColDw1 + kHpm * g);
        float sum[kHpm];
        uint32_t bits[kHpm];
        if (i > 0) {
          tc::tmem_ld8(ta, sum);
          tc::tmem_wait_ld();
        }
#pragma unroll
        for (int k = 0; k < kHpm; ++k) bits[k] = __float_as_uint(fmaf(go[0], act[k], i > 0 ? sum[k] : 0.0f));
        tc::tmem_st8(ta, bits);
      } else {
#pragma unroll
        for (int o = 0; o < kOc; ++o) {
          if (o < oc) {
            float v[kHpm];
#pragma unroll
            for (int k = 0; k < kHpm; ++k) v[k] = go[o] * act[k];
            const float r = warp_reduce_scatter8(v, lane);
            if ((lane & 3) == 0) atomicAdd(s_dw1 + o * kH + kHpm * g + (lane >> 2), r);
          }
        }
      }
    }
    // ---- input rows of the next tile (the MMAs that read the last ones are done) ----
    if (has_in && got) {
      st_split<kFpm, FP32>(tc::taddr(tbase, lb, kColInHi + kFpm * g), tc::taddr(tbase, lb, kColInLo + kFpm * g), e);
      if (g == 0) {
        const float xv[8] = {xn[0], xn[1], xn[2], 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        st_split8<FP32>(tc::taddr(tbase, lb, kColInHi + kXCol), tc::taddr(tbase, lb, kColInLo + kXCol), xv);
      }
    }
    tc::tmem_wait_st();
    tc::fence_proxy_async_smem();
    tc::fence_before_sync();
    if (!__syncthreads_and(got)) {
      ok = false;
      break;
    }
    if (has_in || has_h) {
      if (t == 0) {           // dIN = dH W0 (M=128, N=48, K=64)
        tc::fence_after_sync();
        const uint32_t sbo = (kH / 4) * 128u;
        if (has_h)
          mma_3x(tc::taddr(tbase, 0, par ? kColDin1 : kColDin0), tc::taddr(tbase, 0, kColDhHi), tc::taddr(tbase, 0, kColDhLo),
                 tc::smem_desc(tc::smem_u32(sm + BwdSmem::b2_hi), 128u, sbo),
                 tc::smem_desc(tc::smem_u32(sm + BwdSmem::b2_lo), 128u, sbo), kH / 8, tc::idesc_tf32(kTile, kN2),
                 one_pass);
        tc::mma_commit(bar);
      } else if (t == 32) {   // H = IN W0^T of the next tile (M=128, N=64, K=40)
        tc::fence_after_sync();
        const uint32_t sbo = (kK1 / 4) * 128u;
        if (has_in)
          mma_3x(tc::taddr(tbase, 0, kColH), tc::taddr(tbase, 0, kColInHi), tc::taddr(tbase, 0, kColInLo),
                 tc::smem_desc(tc::smem_u32(sm + BwdSmem::b1_hi), 128u, sbo),
                 tc::smem_desc(tc::smem_u32(sm + BwdSmem::b1_lo), 128u, sbo), kK1 / 8, tc::idesc_tf32(kTile, kH),
                 one_pass);
        tc::mma_commit(bar);
      } else if (t == 64) {   // dW0 += dH^T IN
        tc::fence_after_sync();
        if (has_h) issue_mma3(tbase, sm, i == 0, one_pass);
        tc::mma_commit(bar);
      }
    }
    // ---- next step's loads, under the scatter ----
    x_ptr += 3 * walk.stride;
    if (has_in) {
      const bool live_next = walk.live(i + 2, pt);
      load_grad<kOc>(go_ptr, oc, walk.live(i + 1, pt), gon);
      go_ptr += walk.stride * oc;
      if (load_x) load_point(x_ptr, live_next, xn);
      if constexpr (CACHED) enc_ptr += walk.stride;
      if constexpr (CACHED) load_enc<M>(enc_ptr, a.cap, g, a.active, live_next, en);
    }
    // ---- table-gradient scatter, dL/dx ----
    if (has_din) {
      const PointPair pair = make_pair(xo, lane);
      const uint32_t col_din = par ? kColDin0 : kColDin1;   // the previous step's
      float din[kFpm];
      tc::tmem_ld4(tc::taddr(tbase, lb, col_din + kFpm * g), din);
      tc::tmem_wait_ld();
      if (want_table) {
        float2* gt2 = reinterpret_cast<float2*>(a.grad_table);
#pragma unroll
        for (int i = 0; i < kLpm; ++i) {
          const int l = level_of<M>(g, i);
          if (l < a.active) {
            const float dv[2] = {live_out ? din[2 * i] : 0.0f, live_out ? din[2 * i + 1] : 0.0f};
            scatter_level<2>(a.g, l, pair, dv, live_out, gt2, lane,
                             [](const float f[3], const float d[2], bool x1, int yz) {
                               const float w = corner_weight(f, x1, yz);
                               return make_float2(w * d[0], w * d[1]);
                             });
          }
        }
      }
      if (want_x) {
        float dx[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (g == 0) tc::tmem_ld4(tc::taddr(tbase, lb, col_din + kXCol), dx);
        tc::tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < kLpm; ++i) {
          const int l = level_of<M>(g, i);
          if (l < a.active) {
            float frac[3];
            float2 v[8];
            gather_corners<FP32>(a, l, pair, frac, v);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const float gv = din[2 * i] * v[k].x + din[2 * i + 1] * v[k].y;
#pragma unroll
              for (int d = 0; d < 3; ++d) dx[d] = fmaf(gv, corner_dw(frac, k, d, a.g.lv[l].scale), dx[d]);
            }
          }
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) s_dx[(g * kTile + pt) * 3 + d] = dx[d];
        __syncthreads();
        if (g == 0 && live_out) {
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            float sum = 0.0f;
#pragma unroll
            for (int m = 0; m < M; ++m) sum += s_dx[(m * kTile + pt) * 3 + d];
            a.grad_x[3 * (walk.first + (i - 1) * walk.stride + pt) + d] = sum;
          }
        }
        __syncthreads();
      }
    }
    par ^= 1;
  }
  if (!ok) (void)tc::mbar_wait_bounded(bar, phase ^ 1u);  // drain a timed-out step
  __syncthreads();
  if (!ok && t == 0 && a.status) atomicOr(a.status, SN_STATUS_TIMEOUT);
  tc::fence_after_sync();
  if (ok && walk.count > 0) {
    if constexpr (ONE) {
      float v[kHpm];
      tc::tmem_ld8(tc::taddr(tbase, lb, kColDw1 + kHpm * g), v);
      tc::tmem_wait_ld();
      const float r = warp_reduce_scatter8(v, lane);
      if ((lane & 3) == 0) s_dw1[q * kH + kHpm * g + (lane >> 2)] = r;   // a row a quadrant
    }
    flush_dw0<M>(a, tc::taddr(tbase, lb, kColDw0), reinterpret_cast<float*>(a3));   // (its barriers: all of s_dw1)
    // dW1 (block sums in shared memory)
    for (int e = t; e < oc * kH; e += kNt) {
      double s = (double)s_dw1[e];
      if constexpr (ONE) s = (s + (double)s_dw1[kH + e]) + ((double)s_dw1[2 * kH + e] + (double)s_dw1[3 * kH + e]);
      add_dw1(a, e, s);
    }
  }
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tbase, kBwdCols);
}


// ---------------------------------------------------------------------------
// second-order adjoint of d sdf / d x (SDFNetwork.gradient with create_graph)
// ---------------------------------------------------------------------------
// With IN = [e, x] and Z = [eta, gamma] in the permuted input order (eta = E
// gamma, E = d e / d x), h = IN W0^T + b0 and the sdf row w1 of W1:
//   H = IN W0^T, MU = Z W0^T                                  (first MMAs)
//   u = w1 softplus'(h), delta = MU w1 softplus''(h) + rho w1 softplus'(h)
//   DE = delta W0, VV = u W0 (encoding columns)               (second MMAs)
//   dT_{c,f} += DE_{l,f} w_c + VV_{l,f} (gamma . d w_c / d x)  (scatter)
//   dW0 += delta^T IN + u^T Z over the CTA's points           (third MMAs)
//   db0 += delta (row of ones in IN^T, zero in Z^T),
//   dw1 += MU softplus'(h) + rho softplus(h)  (db1 += rho: column_sums_kernel).
// The third MMAs run in two halves through the same shared-memory operands
// (delta with IN^T, then u with Z^T), each waited for before its operands
// are overwritten.
//
// TMEM columns (512): H [0,64), later DE [0,32); MU [64,128), later VV
// [64,96); IN rows hi/lo [128,208) and Z rows hi/lo [208,288), and after the
// first MMAs delta hi/lo [128,256) and u hi/lo [256,384) (A of the second
// MMAs); dW0 accumulates in [384,432).
constexpr uint32_t kGColH = 0, kGColMu = 64, kGColInHi = 128, kGColInLo = 128 + kK1, kGColZHi = 208,
                   kGColZLo = 208 + kK1, kGColDHi = 128, kGColDLo = 192, kGColUHi = 256, kGColULo = 320,
                   kGColDw0 = 384;
constexpr int kGradMembers = 8;

struct GradSmem {
  static constexpr uint32_t b1_hi = 0, b1_lo = 10240, b2_hi = 20480, b2_lo = 32768, a3 = 45056,
                            b3_hi = a3 + 16 * kSboP, b3_lo = b3_hi + 6 * kSboP, w1 = b3_lo + 6 * kSboP,
                            b0 = w1 + kH * 4, dw1 = b0 + kH * 4, bar = dw1 + 4 * kH * 8,
                            bar3 = bar + 8, slot = bar3 + 8, end = slot + 8;
};
constexpr size_t kGradSmemBytes = GradSmem::end;
static_assert(GradSmem::end <= 227 * 1024, "second-order shared memory map");

// gamma . d w / d x of a corner (the trilinear weight's derivative).
__device__ __forceinline__ float corner_dir_deriv(const float f[3], float s, const float gam[3], bool x1, int yz) {
  const float wx = x1 ? f[0] : 1.0f - f[0], wy = (yz & 1) ? f[1] : 1.0f - f[1], wz = (yz & 2) ? f[2] : 1.0f - f[2];
  const float sx = x1 ? s : -s, sy = (yz & 1) ? s : -s, sz = (yz & 2) ? s : -s;
  return gam[0] * (sx * (wy * wz)) + gam[1] * (sy * (wx * wz)) + gam[2] * (sz * (wx * wy));
}

// Member g's levels of point x: encoding e and eta = E gamma.
template <int M>
__device__ __forceinline__ void encode_eta_group(const FieldArgs& a, int g, bool live, const PointPair& q,
                                                 const float gam[3], float e[2 * (16 / M)],
                                                 float eta[2 * (16 / M)]) {
  constexpr int kLpm = 16 / M;
  const bool any = __any_sync(0xffffffffu, live);
#pragma unroll
  for (int i = 0; i < kLpm; ++i) {
    const int l = level_of<M>(g, i);
    float e0 = 0.0f, e1 = 0.0f, h0 = 0.0f, h1 = 0.0f;
    if (any && l < a.active) {
      float frac[3], w[8], wg[8];
      float2 tv[8];
      gather_corners<true>(a, l, q, frac, tv);
      corner_weights(frac, w);
#pragma unroll
      for (int k = 0; k < 8; ++k) wg[k] = corner_dir_deriv(frac, a.g.lv[l].scale, gam, (k & 1) != 0, k >> 1);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        e0 = __fmaf_rn(w[k], tv[k].x, e0);
        e1 = __fmaf_rn(w[k], tv[k].y, e1);
        h0 = fmaf(wg[k], tv[k].x, h0);
        h1 = fmaf(wg[k], tv[k].y, h1);
      }
    }
    e[2 * i] = live ? e0 : 0.0f;
    e[2 * i + 1] = live ? e1 : 0.0f;
    eta[2 * i] = live ? h0 : 0.0f;
    eta[2 * i + 1] = live ? h1 : 0.0f;
  }
}

// A = [rows hi; rows lo] of a3 (M = 128, K = the tile's points) times B = the
// staged transposed inputs (N = 48) hi and lo, accumulated into dW0.
__device__ __forceinline__ void issue_grad_mma3(uint32_t tbase, const uint8_t* sm, bool fresh, bool one_pass) {
  const uint32_t idesc = tc::idesc_tf32(kTile, kN2);
  const uint32_t d3 = tc::taddr(tbase, 0, kGColDw0);
  const uint64_t da = tc::smem_desc(tc::smem_u32(sm + GradSmem::a3), kLboP, kSboP),
                 dbh = tc::smem_desc(tc::smem_u32(sm + GradSmem::b3_hi), kLboP, kSboP),
                 dbl = tc::smem_desc(tc::smem_u32(sm + GradSmem::b3_lo), kLboP, kSboP);
  for (int ks = 0; ks < kTile / 8; ++ks) {
    const uint64_t k0 = (2u * kLboP * ks) >> 4;
    tc::mma_ss(d3, da + k0, dbh + k0, idesc, (fresh && ks == 0) ? 0u : 1u);
    if (!one_pass) tc::mma_ss(d3, da + k0, dbl + k0, idesc, 1);
  }
}

// Writes v (hi/lo) as row `row` (hi) and row + kH (lo) of a3, column pt.
__device__ __forceinline__ void st_a3(uint8_t* a3, int row, int pt, float v) {
  uint32_t hi, lo;
  tc::tf32_split_even(v, hi, lo);
  st_smem_u32(a3, tc::kmajor_offset_strided(row, pt, kLboP, kSboP), hi);
  st_smem_u32(a3, tc::kmajor_offset_strided(kH + row, pt, kLboP, kSboP), lo);
}
// Writes v (hi/lo) as row `row` of the transposed inputs, column pt.
__device__ __forceinline__ void st_b3(uint8_t* b3_hi, uint8_t* b3_lo, int row, int pt, float v) {
  uint32_t hi, lo;
  tc::tf32_split_even(v, hi, lo);
  const uint32_t off = tc::kmajor_offset_strided(row, pt, kLboP, kSboP);
  st_smem_u32(b3_hi, off, hi);
  st_smem_u32(b3_lo, off, lo);
}

template <int M>
__global__ void __launch_bounds__(128 * M, 1)
field_grad_bwd_tc_kernel(FieldArgs a, const float* __restrict__ gamma, const float* __restrict__ rho_in) {
  constexpr int kNt = 128 * M;
  constexpr int kLpm = 16 / M;
  constexpr int kFpm = 2 * kLpm;
  constexpr int kHpm = kH / M;
  static_assert(kHpm == 8 && kFpm == 4, "eight members per quadrant");
  extern __shared__ __align__(1024) uint8_t sm[];
  float* s_w1 = reinterpret_cast<float*>(sm + GradSmem::w1);
  float* s_b0 = reinterpret_cast<float*>(sm + GradSmem::b0);
  double* s_dw1 = reinterpret_cast<double*>(sm + GradSmem::dw1);   // a row a quadrant
  uint8_t* a3 = sm + GradSmem::a3;
  uint8_t* b3_hi = sm + GradSmem::b3_hi;
  uint8_t* b3_lo = sm + GradSmem::b3_lo;
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + GradSmem::bar);
  uint64_t* bar3 = reinterpret_cast<uint64_t*>(sm + GradSmem::bar3);
  uint32_t* slot = reinterpret_cast<uint32_t*>(sm + GradSmem::slot);
  const int t = threadIdx.x, warp = uniform_warp(), lane = t & 31;
  const int q = warp & 3, g = warp >> 2;
  const int pt = 32 * q + lane;
  const bool want_table = a.grad_table != nullptr;

  stage_w0<M, true>(a, sm + GradSmem::b1_hi, sm + GradSmem::b1_lo, sm + GradSmem::b2_hi, sm + GradSmem::b2_lo);
  if (t < kH) {
    s_w1[t] = a.w1[t];  // the sdf row of W1
    s_b0[t] = a.b0[t];
  }
  // constant rows of the transposed inputs: zeros above the ones row (row
  // kOnesRow is written per tile: one for IN^T, zero for Z^T)
  for (int e = t; e < (kN2 - kOnesRow - 1) * kTile; e += kNt) {
    const int r = kOnesRow + 1 + e / kTile, c = e % kTile;
    const uint32_t off = tc::kmajor_offset_strided(r, c, kLboP, kSboP);
    st_smem_u32(b3_hi, off, 0u);
    st_smem_u32(b3_lo, off, 0u);
  }
  if (warp == 0) {
    tc::tmem_alloc(slot, kBwdCols);
    tc::tmem_relinquish();
  }
  if (t == 0) {
    tc::mbar_init(bar, 1);
    tc::mbar_init(bar3, 1);
  }
  tc::fence_proxy_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = *slot;
  const uint32_t lb = (uint32_t)(32 * q);
  const uint32_t idesc1 = tc::idesc_tf32(kTile, kH), idesc2 = tc::idesc_tf32(kTile, 32);
  const uint32_t sbo1 = (kK1 / 4) * 128u, sbo2 = (kH / 4) * 128u;
  const uint64_t w1_hi = tc::smem_desc(tc::smem_u32(sm + GradSmem::b1_hi), 128u, sbo1),
                 w1_lo = tc::smem_desc(tc::smem_u32(sm + GradSmem::b1_lo), 128u, sbo1),
                 w2_hi = tc::smem_desc(tc::smem_u32(sm + GradSmem::b2_hi), 128u, sbo2),
                 w2_lo = tc::smem_desc(tc::smem_u32(sm + GradSmem::b2_lo), 128u, sbo2);
  const float inv_beta = 1.0f / a.beta;
  uint32_t phase = 0, phase3 = 0;
  bool ok = true, first = true, pending3 = false;
  double dw1 = 0.0;   // of hidden unit kHpm g + lane / 4, over the quadrant's points

  const int64_t n = effective_n(a);
  const int64_t n_tiles = (n + kTile - 1) / kTile;
  float xn[3], gn[3], rn = 0.0f;
  auto load_next = [&](int64_t p) {
    load_point(a, p, n, xn);
    const bool in = p < n;
#pragma unroll
    for (int d = 0; d < 3; ++d) gn[d] = in ? gamma[3 * p + d] : 0.0f;
    rn = (in && rho_in) ? rho_in[p] : 0.0f;
  };
  load_next((int64_t)blockIdx.x * kTile + pt);
  for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int64_t p = tile * kTile + pt;
    const bool live = p < n;
    const float x[3] = {xn[0], xn[1], xn[2]};
    const float gam[3] = {gn[0], gn[1], gn[2]};
    const float rho = rn;
    load_next((tile + gridDim.x) * kTile + pt);
    // ---- IN and Z rows (TMEM, A of the first MMAs), IN^T (B of the third) ----
    float eta[kFpm];
    bool ok3 = true;
    {
      float e[kFpm];
      encode_eta_group<M>(a, g, live, make_pair(x, lane), gam, e, eta);
      st_split<kFpm, true>(tc::taddr(tbase, lb, kGColInHi + kFpm * g), tc::taddr(tbase, lb, kGColInLo + kFpm * g), e);
      st_split<kFpm, true>(tc::taddr(tbase, lb, kGColZHi + kFpm * g), tc::taddr(tbase, lb, kGColZLo + kFpm * g), eta);
      if (g == 0) {
        const float xv[8] = {x[0], x[1], x[2], 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        const float gv[8] = {gam[0], gam[1], gam[2], 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        st_split8<true>(tc::taddr(tbase, lb, kGColInHi + kXCol), tc::taddr(tbase, lb, kGColInLo + kXCol), xv);
        st_split8<true>(tc::taddr(tbase, lb, kGColZHi + kXCol), tc::taddr(tbase, lb, kGColZLo + kXCol), gv);
      }
      // the previous tile's u^T Z MMAs still read a3 and the transposed inputs
      if (pending3) {
        ok3 = tc::mbar_wait_bounded(bar3, phase3);
        if (ok3) {
          phase3 ^= 1u;
          pending3 = false;
        }
      }
#pragma unroll
      for (int i = 0; i < kFpm; ++i) st_b3(b3_hi, b3_lo, kFpm * g + i, pt, e[i]);
      if (g == 0) {
#pragma unroll
        for (int d = 0; d < 3; ++d) st_b3(b3_hi, b3_lo, kXCol + d, pt, x[d]);
        const uint32_t off = tc::kmajor_offset_strided(kOnesRow, pt, kLboP, kSboP);
        st_smem_u32(b3_hi, off, __float_as_uint(1.0f));
        st_smem_u32(b3_lo, off, 0u);
      }
    }
    tc::tmem_wait_st();
    tc::fence_proxy_async_smem();
    tc::fence_before_sync();
    if (!__syncthreads_and(ok3)) {
      ok = false;
      break;
    }
    if (t == 0) {  // H = IN W0^T, MU = Z W0^T (M=128, N=64, K=40)
      tc::fence_after_sync();
      mma_3x(tc::taddr(tbase, 0, kGColH), tc::taddr(tbase, 0, kGColInHi), tc::taddr(tbase, 0, kGColInLo), w1_hi,
             w1_lo, kK1 / 8, idesc1);
      mma_3x(tc::taddr(tbase, 0, kGColMu), tc::taddr(tbase, 0, kGColZHi), tc::taddr(tbase, 0, kGColZLo), w1_hi,
             w1_lo, kK1 / 8, idesc1);
      tc::mma_commit(bar);
    }
    bool got = tc::mbar_wait_bounded(bar, phase);
    phase ^= 1u;
    if (!__syncthreads_and(got)) {
      ok = false;
      break;
    }
    tc::fence_after_sync();
    // ---- u, delta, dw1 for this member's hidden units 8g .. 8g + 7 ----
    float u[kHpm];
    {
      float h[kHpm], mu[kHpm];
      tc::tmem_ld8(tc::taddr(tbase, lb, kGColH + kHpm * g), h);
      tc::tmem_ld8(tc::taddr(tbase, lb, kGColMu + kHpm * g), mu);
      tc::tmem_wait_ld();
      float dl[kHpm], v[kHpm];
#pragma unroll
      for (int i = 0; i < kHpm; ++i) {
        const int j = kHpm * g + i;
        const float pre = h[i] + s_b0[j];
        float act, s1;
        softplus_fwd_grad_fast(pre, a.beta, inv_beta, a.thresh, act, s1);
        const float s2 = pre * a.beta > a.thresh ? 0.0f : a.beta * s1 * (1.0f - s1);
        const float w1 = s_w1[j];
        u[i] = live ? w1 * s1 : 0.0f;
        dl[i] = live ? fmaf(mu[i] * w1, s2, rho * w1 * s1) : 0.0f;
        v[i] = live ? fmaf(mu[i], s1, rho * act) : 0.0f;
      }
      dw1 += (double)warp_reduce_scatter8(v, lane);
      st_split8<true>(tc::taddr(tbase, lb, kGColDHi + kHpm * g), tc::taddr(tbase, lb, kGColDLo + kHpm * g), dl);
      st_split8<true>(tc::taddr(tbase, lb, kGColUHi + kHpm * g), tc::taddr(tbase, lb, kGColULo + kHpm * g), u);
#pragma unroll
      for (int i = 0; i < kHpm; ++i) st_a3(a3, kHpm * g + i, pt, dl[i]);
    }
    tc::tmem_wait_st();
    tc::fence_proxy_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    if (t == 0) {  // DE = delta W0, VV = u W0 (M=128, N=32 encoding columns, K=64)
      tc::fence_after_sync();
      mma_3x(tc::taddr(tbase, 0, kGColH), tc::taddr(tbase, 0, kGColDHi), tc::taddr(tbase, 0, kGColDLo), w2_hi,
             w2_lo, kH / 8, idesc2);
      mma_3x(tc::taddr(tbase, 0, kGColMu), tc::taddr(tbase, 0, kGColUHi), tc::taddr(tbase, 0, kGColULo), w2_hi,
             w2_lo, kH / 8, idesc2);
      tc::mma_commit(bar);
    }
    got = tc::mbar_wait_bounded(bar, phase);
    phase ^= 1u;
    if (!__syncthreads_and(got)) {
      ok = false;
      break;
    }
    tc::fence_after_sync();
    if (t == 32) {  // dW0 += delta^T IN (db0 from the ones row), behind the second MMAs
      issue_grad_mma3(tbase, sm, first, false);
      tc::mma_commit(bar3);
    }
    first = false;
    pending3 = true;
    // ---- table gradient for this member's levels ----
    if (want_table) {
      float de[kFpm], vv[kFpm];
      tc::tmem_ld4(tc::taddr(tbase, lb, kGColH + kFpm * g), de);
      tc::tmem_ld4(tc::taddr(tbase, lb, kGColMu + kFpm * g), vv);
      tc::tmem_wait_ld();
      float2* gt2 = reinterpret_cast<float2*>(a.grad_table);
      const PointPair pair = make_pair(x, lane);
#pragma unroll
      for (int i = 0; i < kLpm; ++i) {
        const int l = level_of<M>(g, i);
        if (l < a.active) {
          const float sc = a.g.lv[l].scale;
          const float dv[7] = {live ? de[2 * i] : 0.0f, live ? de[2 * i + 1] : 0.0f, live ? vv[2 * i] : 0.0f,
                               live ? vv[2 * i + 1] : 0.0f, gam[0], gam[1], gam[2]};
          scatter_level<7>(a.g, l, pair, dv, live, gt2, lane, [sc](const float f[3], const float d[7], bool x1, int yz) {
            const float w = corner_weight(f, x1, yz), wg = corner_dir_deriv(f, sc, d + 4, x1, yz);
            return make_float2(fmaf(d[0], w, d[2] * wg), fmaf(d[1], w, d[3] * wg));
          });
        }
      }
    }
    // ---- dW0 += u^T Z: wait for delta^T IN, then reuse its operands ----
    ok3 = tc::mbar_wait_bounded(bar3, phase3);
    if (ok3) {
      phase3 ^= 1u;
      pending3 = false;
    }
    if (ok3) {
#pragma unroll
      for (int i = 0; i < kHpm; ++i) st_a3(a3, kHpm * g + i, pt, u[i]);
#pragma unroll
      for (int i = 0; i < kFpm; ++i) st_b3(b3_hi, b3_lo, kFpm * g + i, pt, eta[i]);
      if (g == 0) {
#pragma unroll
        for (int d = 0; d < 3; ++d) st_b3(b3_hi, b3_lo, kXCol + d, pt, gam[d]);
        const uint32_t off = tc::kmajor_offset_strided(kOnesRow, pt, kLboP, kSboP);
        st_smem_u32(b3_hi, off, 0u);
        st_smem_u32(b3_lo, off, 0u);
      }
    }
    tc::fence_proxy_async_smem();
    tc::fence_before_sync();
    if (!__syncthreads_and(ok3)) {
      ok = false;
      break;
    }
    if (t == 32) {
      tc::fence_after_sync();
      issue_grad_mma3(tbase, sm, false, false);
      tc::mma_commit(bar3);
    }
    pending3 = true;
  }
  if (!ok) (void)tc::mbar_wait_bounded(bar, phase ^ 1u);  // drain a timed-out first/second MMA
  if (pending3) ok = tc::mbar_wait_bounded(bar3, phase3) && ok;
  ok = __syncthreads_and(ok);
  if (!ok && t == 0 && a.status) atomicOr(a.status, SN_STATUS_TIMEOUT);
  tc::fence_after_sync();
  if (ok && !first) {
    if ((lane & 3) == 0) s_dw1[q * kH + kHpm * g + (lane >> 2)] = dw1;
    flush_dw0<M>(a, tc::taddr(tbase, lb, kGColDw0), reinterpret_cast<float*>(a3));   // (its barriers: all of s_dw1)
    if (t < kH) add_dw1(a, t, (s_dw1[t] + s_dw1[kH + t]) + (s_dw1[2 * kH + t] + s_dw1[3 * kH + t]));
  }
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tbase, kBwdCols);
}

// ---------------------------------------------------------------------------
// d sdf / d x (SDFNetwork.gradient): sdf and grad = W0x^T u + E^T (W0e^T u)
// ---------------------------------------------------------------------------
// H = IN W0^T (first MMA), u = w1 softplus'(H + b0), sdf = w1 . softplus + b1,
// V = u W0 (second MMA, all 48 input columns), and per point
// grad = V_x + sum over levels and corners of (V_{l,0} T_{c,0} + V_{l,1} T_{c,1}) d w_c / d x.
// TMEM columns (256, two CTAs per SM): H [0,64); IN rows hi/lo [64,144), after
// the first MMA u hi/lo [64,192) (A of the second); V [192,240).
constexpr uint32_t kFColH = 0, kFColInHi = 64, kFColInLo = 64 + kK1, kFColUHi = 64, kFColULo = 128,
                   kFColV = 192;
constexpr int kGradFwdMembers = 4;

template <int M>
struct GradFwdSmem {
  static constexpr uint32_t b1_hi = 0, b1_lo = 10240, b2_hi = 20480, b2_lo = 32768, w1 = 45056, b0 = w1 + kH * 4,
                            part = b0 + kH * 4, bar = part + M * kTile * 16, slot = bar + 8, end = slot + 8;
  // more than 228/3 KB, so at most two CTAs (2 x 256 TMEM columns) per SM
  static constexpr size_t bytes = 80 * 1024;
};
static_assert(GradFwdSmem<kGradFwdMembers>::end <= GradFwdSmem<kGradFwdMembers>::bytes, "gradient shared memory map");

template <int M>
__global__ void __launch_bounds__(128 * M, 2)
field_grad_fwd_tc_kernel(FieldArgs a, float* __restrict__ out_sdf, float* __restrict__ out_grad) {
  constexpr int kLpm = 16 / M;
  constexpr int kFpm = 2 * kLpm;
  constexpr int kHpm = kH / M;
  static_assert(kFpm == 8 && kHpm == 16, "four members per quadrant");
  using Sm = GradFwdSmem<M>;
  extern __shared__ __align__(1024) uint8_t sm[];
  float* s_w1 = reinterpret_cast<float*>(sm + Sm::w1);
  float* s_b0 = reinterpret_cast<float*>(sm + Sm::b0);
  float4* s_part = reinterpret_cast<float4*>(sm + Sm::part);
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + Sm::bar);
  uint32_t* slot = reinterpret_cast<uint32_t*>(sm + Sm::slot);
  const int t = threadIdx.x, warp = uniform_warp(), lane = t & 31;
  const int q = warp & 3, g = warp >> 2;
  const int pt = 32 * q + lane;

  stage_w0<M, true>(a, sm + Sm::b1_hi, sm + Sm::b1_lo, sm + Sm::b2_hi, sm + Sm::b2_lo);
  if (t < kH) {
    s_w1[t] = a.w1[t];  // the sdf row of W1
    s_b0[t] = a.b0[t];
  }
  const float b1v = a.b1[0];
  if (warp == 0) {
    tc::tmem_alloc(slot, kCols);
    tc::tmem_relinquish();
  }
  if (t == 0) tc::mbar_init(bar, 1);
  tc::fence_proxy_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tbase = *slot;
  const uint32_t lb = (uint32_t)(32 * q);
  const uint32_t idesc1 = tc::idesc_tf32(kTile, kH), idesc2 = tc::idesc_tf32(kTile, kN2);
  const uint32_t sbo1 = (kK1 / 4) * 128u, sbo2 = (kH / 4) * 128u;
  const uint64_t w1_hi = tc::smem_desc(tc::smem_u32(sm + Sm::b1_hi), 128u, sbo1),
                 w1_lo = tc::smem_desc(tc::smem_u32(sm + Sm::b1_lo), 128u, sbo1),
                 w2_hi = tc::smem_desc(tc::smem_u32(sm + Sm::b2_hi), 128u, sbo2),
                 w2_lo = tc::smem_desc(tc::smem_u32(sm + Sm::b2_lo), 128u, sbo2);
  const float inv_beta = 1.0f / a.beta;
  uint32_t phase = 0;
  bool ok = true;

  const int64_t n = effective_n(a);
  const int64_t n_tiles = (n + kTile - 1) / kTile;
  float xn[3];
  load_point(a, (int64_t)blockIdx.x * kTile + pt, n, xn);
  for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int64_t p = tile * kTile + pt;
    const bool live = p < n;
    const float x[3] = {xn[0], xn[1], xn[2]};
    load_point(a, (tile + gridDim.x) * kTile + pt, n, xn);
    {
      float e[kFpm];
      encode_group<M>(a, g, live, make_pair(x, lane), e);
      st_split<kFpm>(tc::taddr(tbase, lb, kFColInHi + kFpm * g), tc::taddr(tbase, lb, kFColInLo + kFpm * g), e);
      if (g == 0) {
        const float xv[8] = {x[0], x[1], x[2], 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        st_split8(tc::taddr(tbase, lb, kFColInHi + kXCol), tc::taddr(tbase, lb, kFColInLo + kXCol), xv);
      }
    }
    tc::tmem_wait_st();
    tc::fence_before_sync();
    __syncthreads();
    if (t == 0) {  // H = IN W0^T (M=128, N=64, K=40)
      tc::fence_after_sync();
      mma_3x(tc::taddr(tbase, 0, kFColH), tc::taddr(tbase, 0, kFColInHi), tc::taddr(tbase, 0, kFColInLo), w1_hi,
             w1_lo, kK1 / 8, idesc1);
      tc::mma_commit(bar);
    }
    bool got = tc::mbar_wait_bounded(bar, phase);
    phase ^= 1u;
    if (!__syncthreads_and(got)) {
      ok = false;
      break;
    }
    tc::fence_after_sync();
    // u and the sdf partial for hidden units kHpm g .. kHpm g + kHpm - 1
    float sdf_part = 0.0f;
    {
      float h[kHpm], u[kHpm];
      tc::tmem_ld16(tc::taddr(tbase, lb, kFColH + kHpm * g), h);
      tc::tmem_wait_ld();
#pragma unroll
      for (int i = 0; i < kHpm; ++i) {
        const int j = kHpm * g + i;
        float act, s1;
        softplus_fwd_grad_fast(h[i] + s_b0[j], a.beta, inv_beta, a.thresh, act, s1);
        u[i] = s_w1[j] * s1;
        sdf_part = fmaf(s_w1[j], act, sdf_part);
      }
      st_split<kHpm>(tc::taddr(tbase, lb, kFColUHi + kHpm * g), tc::taddr(tbase, lb, kFColULo + kHpm * g), u);
    }
    tc::tmem_wait_st();
    tc::fence_before_sync();
    __syncthreads();
    if (t == 0) {  // V = u W0 (M=128, N=48, K=64)
      tc::fence_after_sync();
      mma_3x(tc::taddr(tbase, 0, kFColV), tc::taddr(tbase, 0, kFColUHi), tc::taddr(tbase, 0, kFColULo), w2_hi,
             w2_lo, kH / 8, idesc2);
      tc::mma_commit(bar);
    }
    got = tc::mbar_wait_bounded(bar, phase);
    phase ^= 1u;
    if (!__syncthreads_and(got)) {
      ok = false;
      break;
    }
    tc::fence_after_sync();
    // gradient partial: this member's levels (+ the linear x part for member 0)
    {
      float v[kFpm], vx[8];
      tc::tmem_ld8(tc::taddr(tbase, lb, kFColV + kFpm * g), v);
      tc::tmem_ld8(tc::taddr(tbase, lb, kFColV + kXCol), vx);
      tc::tmem_wait_ld();
      float gx[3] = {0.0f, 0.0f, 0.0f};
      if (g == 0) {
        gx[0] = vx[0];
        gx[1] = vx[1];
        gx[2] = vx[2];
      }
      if (__any_sync(0xffffffffu, live)) {
        const PointPair pp = make_pair(x, lane);
#pragma unroll
        for (int i = 0; i < kLpm; ++i) {
          const int l = level_of<M>(g, i);
          if (l < a.active) {
            float frac[3];
            float2 tv[8];
            gather_corners<true>(a, l, pp, frac, tv);
            const float s = a.g.lv[l].scale;
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const float gk = v[2 * i] * tv[k].x + v[2 * i + 1] * tv[k].y;
#pragma unroll
              for (int d = 0; d < 3; ++d) gx[d] = fmaf(gk, corner_dw(frac, k, d, s), gx[d]);
            }
          }
        }
      }
      s_part[g * kTile + pt] = make_float4(sdf_part, gx[0], gx[1], gx[2]);
    }
    __syncthreads();
    // (the next tile writes s_part only after two more barriers)
    if (g == 0 && live) {
      float4 s = s_part[pt];
#pragma unroll
      for (int m = 1; m < M; ++m) {
        const float4 o = s_part[m * kTile + pt];
        s.x += o.x;
        s.y += o.y;
        s.z += o.z;
        s.w += o.w;
      }
      if (out_sdf) out_sdf[p] = s.x + b1v;
      out_grad[3 * p + 0] = s.y;
      out_grad[3 * p + 1] = s.z;
      out_grad[3 * p + 2] = s.w;
    }
  }
  if (!ok) {
    if (t == 0 && a.status) atomicOr(a.status, SN_STATUS_TIMEOUT);
    (void)tc::mbar_wait_bounded(bar, phase ^ 1u);
  }
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tbase, kCols);
}

// The bounded mbarrier wait of the tensor-core kernels, on an mbarrier that
// nothing arrives at, for `polls` polls (0: the kernels' own limit): the wait
// gives up and the timeout is reported through the status word, as a kernel
// whose MMAs never completed reports it.  The kernel then returns normally.
__global__ void bounded_wait_selftest_kernel(int32_t* status, uint32_t polls) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) tc::mbar_init(&bar, 1);
  __syncthreads();
  const bool got = tc::mbar_wait_polls(&bar, 0, polls ? polls : tc::kWaitLimit);
  if (!got && threadIdx.x == 0) atomicOr(status, SN_STATUS_TIMEOUT);
}

}  // namespace

int bounded_wait_selftest(int32_t* status, uint32_t polls, cudaStream_t st) {
  bounded_wait_selftest_kernel<<<1, 32, 0, st>>>(status, polls);
  return check_launch("bounded_wait_selftest");
}
uint32_t bounded_wait_limit() { return tc::kWaitLimit; }

// Launchers used by sn_field_fwd / sn_field_bwd (field.cu).
int field_fwd_tc_segments(const FieldArgs* segs, int n_seg, cudaStream_t st) {
  constexpr int M = kFwdMembers;
  SN_REQUIRE(n_seg >= 1 && n_seg <= kMaxSegments, "field_fwd: %d segments (1..%d)", n_seg, kMaxSegments);
  const bool one = segs[0].out_cols == 1;
  FieldSegments fs;
  memset(&fs, 0, sizeof(fs));
  fs.n = n_seg;
  int64_t max_tiles = 0;
  bool fp32 = true;
  for (int i = 0; i < n_seg; ++i) {
    fp32 = fp32 && !segs[i].table_half && !segs[i].one_pass && !segs[i].bf16;
    SN_REQUIRE((segs[i].out_cols == 1) == one, "field_fwd: segments mix one and several output columns");
    fs.seg[i] = segs[i];
    const int64_t tiles = (segs[i].cap + kTile - 1) / kTile;
    if (tiles > max_tiles) max_tiles = tiles;
  }
  // the precision as a template argument: without its branches at every level the FP32
  // forward of a 256^3 lattice takes 3.30 ms instead of 3.51
  const auto fn = one ? (fp32 ? field_fwd_tc_kernel<true, M, true> : field_fwd_tc_kernel<true, M, false>)
                      : (fp32 ? field_fwd_tc_kernel<false, M, true> : field_fwd_tc_kernel<false, M, false>);
  const size_t smem = one ? FwdSmem<M>::bytes<true> : FwdSmem<M>::bytes<false>;
  SN_TRY(ensure_smem_limit(reinterpret_cast<const void*>(fn), smem, "field_fwd"));
  const int64_t cap = (M == 4 ? 2LL : 1LL) * num_sms();
  const unsigned grid = (unsigned)(max_tiles < cap ? (max_tiles > 0 ? max_tiles : 1) : cap);
  launch_chained(fn, grid, 128 * M, smem, st, fs);
  return check_launch("field_fwd");
}

int field_fwd_tc(const FieldArgs& a, cudaStream_t st) { return field_fwd_tc_segments(&a, 1, st); }

int field_grad_fwd_tc(const FieldArgs& a, float* sdf, float* grad, cudaStream_t st) {
  constexpr int M = kGradFwdMembers;
  constexpr size_t smem = GradFwdSmem<M>::bytes;
  const void* fn = reinterpret_cast<const void*>(field_grad_fwd_tc_kernel<M>);
  SN_TRY(ensure_smem_limit(fn, smem, "field_grad_fwd"));
  const int64_t n_tiles = (a.cap + kTile - 1) / kTile;
  const int64_t cap = 2LL * num_sms();
  const unsigned grid = (unsigned)(n_tiles < cap ? n_tiles : cap);
  field_grad_fwd_tc_kernel<M><<<grid, 128 * M, smem, st>>>(a, sdf, grad);
  return check_launch("field_grad_fwd");
}

int field_grad_bwd_tc(const FieldArgs& a, const float* gamma, const float* rho, cudaStream_t st) {
  constexpr int M = kGradMembers;
  const void* fn = reinterpret_cast<const void*>(field_grad_bwd_tc_kernel<M>);
  SN_TRY(ensure_smem_limit(fn, kGradSmemBytes, "field_grad_bwd"));
  const int64_t n_tiles = (a.cap + kTile - 1) / kTile;
  const int64_t cap = num_sms();
  const unsigned grid = (unsigned)(n_tiles < cap ? n_tiles : cap);
  field_grad_bwd_tc_kernel<M><<<grid, 128 * M, kGradSmemBytes, st>>>(a, gamma, rho);
  return check_launch("field_grad_bwd");
}

template <bool ONE, bool CACHED, bool DX, bool FP32>
static int launch_bwd(const FieldArgs& a, cudaStream_t st) {
  const auto fn = field_bwd_tc_kernel<ONE, kBwdMembers, CACHED, DX, FP32>;
  SN_TRY(ensure_smem_limit(reinterpret_cast<const void*>(fn), kBwdSmemBytes, "field_bwd"));
  const int64_t n_tiles = (a.cap + kTile - 1) / kTile;
  const int64_t cap = num_sms();
  launch_chained(fn, (unsigned)(n_tiles < cap ? n_tiles : cap), 128 * kBwdMembers, kBwdSmemBytes, st, a);
  return check_launch("field_bwd");
}
template <bool ONE, bool DX, bool FP32>
static int launch_bwd(const FieldArgs& a, cudaStream_t st) {
  return a.enc_in ? launch_bwd<ONE, true, DX, FP32>(a, st) : launch_bwd<ONE, false, DX, FP32>(a, st);
}
// The training calls (one output, FP32) without their branches; the others decide
// at run time what they are asked for.
int field_bwd_tc(const FieldArgs& a, cudaStream_t st) {
  if (a.out_cols != 1) return launch_bwd<false, true, false>(a, st);
  if (a.table_half || a.one_pass) return launch_bwd<true, true, false>(a, st);
  return a.grad_x ? launch_bwd<true, true, true>(a, st) : launch_bwd<true, false, true>(a, st);
}

}  // namespace sn
