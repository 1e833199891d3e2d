// Definitions shared by the standalone encoding kernels (field.cu) and the
// tensor-core field kernels (field_tc.cu): hash-grid
// level geometry in tiny-cuda-nn's conventions (see field.cu), the 8-corner
// lookup of one level, and the argument block of the fused field kernels.
#pragma once

#include "common.cuh"

namespace sn {

constexpr int kH = 64;                    // hidden width (fixed, models/fields.py conf d_hidden)
constexpr int kMaxL = 16;                 // levels handled by the fused kernels
constexpr int kF = 2;                     // features per level (SuperNormal hard-codes 2)
constexpr int kDinMax = 3 + kMaxL * kF;   // 35
constexpr int kDinPad = 36;               // row stride of W0 in shared memory
constexpr int kDoutMax = 16;

// Index arithmetic of a level: a masked XOR hash; a dense index whose corner
// differences are below the level size (so one modulo serves four corners);
// anything else, one modulo per corner.
enum LevelKind : uint32_t { kHashed = 0, kDense = 1, kGeneralDense = 2, kGeneralHash = 3 };

// One level, as two 16-byte loads from the kernel parameters.
struct __align__(16) LevelDev {
  float scale;
  uint32_t offset;  // first entry
  uint32_t size;    // entries in the level (tcnn hashmap_size)
  uint32_t kind;    // LevelKind
  uint32_t my, mz;  // factors of y and z: the dense strides or the hash primes
  uint32_t magic;   // Granlund-Montgomery reciprocal of size
  uint32_t shifts;  // its two shifts, low bytes first
};
struct GridDev {
  int L;
  LevelDev lv[kMaxL];
};

// n mod d for uint32 n and invariant d (Granlund & Montgomery 1994, fig. 4.1).
__device__ __forceinline__ uint32_t fast_mod(uint32_t n, uint32_t d, uint32_t m, int s1, int s2) {
  const uint32_t t = __umulhi(m, n);
  const uint32_t q = (t + ((n - t) >> s1)) >> s2;
  return n - q * d;
}

struct LevelCorners {
  uint32_t idx[8];
  float w[8];
  float frac[3];
  uint32_t cell[3];  // integer cell coordinates (the 8 indices are a function of these)
};

__device__ __forceinline__ uint32_t level_mod(const LevelDev& v, uint32_t n) {
  return fast_mod(n, v.size, v.magic, v.shifts & 0xffu, v.shifts >> 8);
}

// Index within the level of the corner with integer coordinates (x, y, z).
__device__ __forceinline__ uint32_t corner_at(const LevelDev& v, uint32_t x, uint32_t y, uint32_t z) {
  const uint32_t ty = y * v.my, tz = z * v.mz;
  if (v.kind == kHashed) return (x ^ ty ^ tz) & (v.size - 1u);
  return level_mod(v, v.kind == kGeneralHash ? x ^ ty ^ tz : x + ty + tz);
}

// Indices within the level of the four corners (x, y + (j & 1), z + (j >> 1)).
// A branch per level (the same on every lane) instead of selects per corner, and
// one modulo for the four corners of a dense level: they lie d < size above the
// first, so they are (first mod size) + d less at most one size, or, where the
// uint32 index wraps between them (cells around the origin), the wrapped index
// itself, which is below d.
__device__ __forceinline__ void corner_quad(const LevelDev& v, uint32_t x, uint32_t y, uint32_t z,
                                            uint32_t idx[4]) {
  const uint32_t y0 = y * v.my, z0 = z * v.mz;
  if (v.kind == kHashed) {
    const uint32_t y1 = y0 + v.my, z1 = z0 + v.mz, m = v.size - 1u;
    idx[0] = (x ^ (y0 ^ z0)) & m;
    idx[1] = (x ^ (y1 ^ z0)) & m;
    idx[2] = (x ^ (y0 ^ z1)) & m;
    idx[3] = (x ^ (y1 ^ z1)) & m;
  } else if (v.kind == kDense) {
    const uint32_t u = x + y0 + z0;
    const uint32_t d[4] = {0u, v.my, v.mz, v.my + v.mz};
    // size >= 2: the first shift is one
    const uint32_t t = __umulhi(v.magic, u);
    idx[0] = u - ((t + ((u - t) >> 1)) >> (v.shifts >> 8)) * v.size;
#pragma unroll
    for (int j = 1; j < 4; ++j) {
      const uint32_t w = u + d[j], r = idx[0] + d[j];
      idx[j] = w < u ? w : min(r, r - v.size);
    }
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) idx[j] = corner_at(v, x, y + (j & 1), z + (j >> 1));
  }
}

// Trilinear weights of the 8 corners from the cell fractions, (wx * wy) * wz.
__device__ __forceinline__ void corner_weights(const float frac[3], float w[8]) {
  float w0[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) w0[d] = __fsub_rn(1.0f, frac[d]);
  float wxy[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) wxy[k] = __fmul_rn((k & 1) ? frac[0] : w0[0], (k & 2) ? frac[1] : w0[1]);
#pragma unroll
  for (int k = 0; k < 8; ++k) w[k] = __fmul_rn(wxy[k & 3], (k & 4) ? frac[2] : w0[2]);
}

// The 8 corners of x's cell at level l: entry indices and trilinear weights.
// Per-dimension terms are formed once (index of corner (dx,dy,dz) = a sum of
// the dense strides or an XOR of the prime products, weight = (wx * wy) * wz),
// which gives exactly the values of the corner-by-corner formula.
__device__ __forceinline__ void level_corners(const GridDev& g, int l, const float x[3],
                                              LevelCorners& c) {
  const LevelDev lv = g.lv[l];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float p = __fmaf_rn(lv.scale, x[d], 0.5f);
    const float f = floorf(p);
    c.cell[d] = (uint32_t)(int)f;
    c.frac[d] = __fsub_rn(p, f);
  }
  uint32_t i0[4], i1[4];
  corner_quad(lv, c.cell[0], c.cell[1], c.cell[2], i0);
  corner_quad(lv, c.cell[0] + 1u, c.cell[1], c.cell[2], i1);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    c.idx[2 * j] = lv.offset + i0[j];
    c.idx[2 * j + 1] = lv.offset + i1[j];
  }
  corner_weights(c.frac, c.w);
}

// d w_k / d x_d for linear interpolation (scale * +-1 * product of the other two factors).
__device__ __forceinline__ float corner_dw(const float frac[3], int k, int d, float s) {
  float w = 1.0f;
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    if (e == d) continue;
    const bool hi = (k >> e) & 1;
    w *= hi ? frac[e] : 1.0f - frac[e];
  }
  return ((k >> d) & 1) ? s * w : -s * w;
}

__device__ __forceinline__ void encode_level(const float* __restrict__ table, const GridDev& g,
                                             int l, const float x[3], float& e0, float& e1) {
  LevelCorners c;
  level_corners(g, l, x, c);
  const float2* t2 = reinterpret_cast<const float2*>(table);
  float2 v[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) v[k] = __ldg(t2 + c.idx[k]);
  float a = 0.0f, b = 0.0f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    a = __fmaf_rn(c.w[k], v[k].x, a);
    b = __fmaf_rn(c.w[k], v[k].y, b);
  }
  e0 = a;
  e1 = b;
}

struct FieldArgs {
  int64_t cap;
  const int32_t* count;   // optional device count (n = min(*count, cap))
  const float* x;
  const float* table;
  GridDev g;
  int active;             // active levels
  int din;                // 3 + L*F
  int dout;               // rows of W1
  int out_cols;           // outputs computed / gradients read (<= dout)
  float beta, thresh;
  const float* w0;        // (64, din)
  const float* b0;        // (64)
  const float* w1;        // (dout, 64)
  const float* b1;        // (dout)
  float* out;             // (n, out_cols)
  const float* grad_out;  // (n, out_cols)
  float* grad_table;
  float* grad_w0;
  float* grad_b0;
  float* grad_w1;
  double* w1_sums;        // optional: the weight gradient of layer 1 goes there instead of grad_w1
  float* grad_x;          // (n, 3) optional
  int32_t* status;        // optional: SN_STATUS_TIMEOUT is OR-ed here
  bool table_half;        // table holds FP16 pairs (SN_FIELD_TABLE_FP16)
  bool one_pass;          // single-pass TF32 MLP products (SN_FIELD_MLP_TF32)
  bool bf16;              // forward: single-pass BF16 first layer (SN_FIELD_MLP_BF16)
  float2* enc_out;        // forward: level l of point p written at enc_out[l * cap + p]
  const float2* enc_in;   // backward: the encoding read from there instead of gathered
};

// The points of two neighbouring lanes (2i, 2i + 1): a is the even lane's.
struct PointPair {
  float a[3], b[3];
  uint32_t odd;  // this lane is the odd one
};
__device__ __forceinline__ PointPair make_pair(const float x[3], int lane) {
  PointPair q;
  q.odd = (uint32_t)lane & 1u;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float o = __shfl_xor_sync(0xffffffffu, x[d], 1);
    q.a[d] = q.odd ? o : x[d];
    q.b[d] = q.odd ? x[d] : o;
  }
  return q;
}

// The 8 corner entries of this lane's point at level l, and its cell fractions.
// Reached by all 32 lanes of a warp at the same level.
//
// A warp's gather costs the L1 one wavefront per 128-byte line that its lanes
// touch, and with every lane loading its own eight corners that bounds the
// encoding (77 % of the L1 data pipe's peak on the SDF lattice).  The two x
// corners of a cell lie in one line 15 times out of 16 (entries differ in their
// low index bits only), so here two lanes load one point's two x corners
// together: the even lane the x side 0 and the odd lane side 1 of the even
// lane's point, then side 1 and side 0 of the odd lane's.  Either lane then
// has its own side 0 and gets side 1 by a shuffle: eight loads a lane as
// before, half the lines.  256^3 SDF lattice: 5.55 -> 5.02 ms (by itself); the values
// and their order of summation are unchanged.
// FP32: the table is known to be FP32 (no branch on it at every level).
template <bool FP32 = false>
__device__ __forceinline__ void gather_corners(const FieldArgs& a, int l, const PointPair& q, float frac[3],
                                               float2 v[8]) {
  const LevelDev lv = a.g.lv[l];
  const float s = lv.scale;
  uint32_t ca[3], cb[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float pa = __fmaf_rn(s, q.a[d], 0.5f), pb = __fmaf_rn(s, q.b[d], 0.5f);
    const float own = q.odd ? pb : pa;
    frac[d] = __fsub_rn(own, floorf(own));
    ca[d] = (uint32_t)__float2int_rd(pa);
    cb[d] = (uint32_t)__float2int_rd(pb);
  }
  uint32_t ia[4], ib[4];
  corner_quad(lv, ca[0] + q.odd, ca[1], ca[2], ia);
  corner_quad(lv, cb[0] + (q.odd ^ 1u), cb[1], cb[2], ib);
  if (!FP32 && a.table_half) {
    const uint32_t* t = reinterpret_cast<const uint32_t*>(a.table) + lv.offset;
    uint32_t va[4], vb[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      va[j] = __ldg(t + ia[j]);
      vb[j] = __ldg(t + ib[j]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t own = q.odd ? vb[j] : va[j];
      const uint32_t other = __shfl_xor_sync(0xffffffffu, q.odd ? va[j] : vb[j], 1);
      v[2 * j] = __half22float2(*reinterpret_cast<const __half2*>(&own));
      v[2 * j + 1] = __half22float2(*reinterpret_cast<const __half2*>(&other));
    }
  } else {
    const float2* t = reinterpret_cast<const float2*>(a.table) + lv.offset;
    float2 va[4], vb[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      va[j] = __ldg(t + ia[j]);
      vb[j] = __ldg(t + ib[j]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      v[2 * j] = q.odd ? vb[j] : va[j];
      v[2 * j + 1].x = __shfl_xor_sync(0xffffffffu, q.odd ? va[j].x : vb[j].x, 1);
      v[2 * j + 1].y = __shfl_xor_sync(0xffffffffu, q.odd ? va[j].y : vb[j].y, 1);
    }
  }
}

// Encoding of this lane's point at one level (all 32 lanes of a warp together).
template <bool FP32>
__device__ __forceinline__ void encode_level_pair(const FieldArgs& a, int l, const PointPair& q, float& e0,
                                                  float& e1) {
  float frac[3], w[8];
  float2 v[8];
  gather_corners<FP32>(a, l, q, frac, v);
  corner_weights(frac, w);
  float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    s0 = __fmaf_rn(w[k], v[k].x, s0);
    s1 = __fmaf_rn(w[k], v[k].y, s1);
  }
  e0 = s0;
  e1 = s1;
}

__device__ __forceinline__ int64_t effective_n(const FieldArgs& a) {
  if (!a.count) return a.cap;
  const int64_t c = *a.count;
  return c < a.cap ? c : a.cap;
}

// Tensor-core launchers (field_tc.cu).
int field_fwd_tc(const FieldArgs& a, cudaStream_t st);
int field_fwd_tc_segments(const FieldArgs* segs, int n_seg, cudaStream_t st);
int field_bwd_tc(const FieldArgs& a, cudaStream_t st);
int bounded_wait_selftest(int32_t* status, uint32_t polls, cudaStream_t st);
uint32_t bounded_wait_limit();
int field_grad_fwd_tc(const FieldArgs& a, float* sdf, float* grad, cudaStream_t st);
int field_grad_bwd_tc(const FieldArgs& a, const float* gamma, const float* rho, cudaStream_t st);

// Host helpers (field.cu).
int make_grid_dev(const sn_grid_desc* d, GridDev& g);
int fill_field_args(FieldArgs& a, int64_t n, const int32_t* count, const float* x, const float* table,
                    const sn_grid_desc* grid, int active_levels, const sn_mlp_desc* mlp, int out_cols);

}  // namespace sn
