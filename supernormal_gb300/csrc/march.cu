// Occupancy-grid ray marching, sample packing and grid queries.
//
// The marcher restates nerfacc's fixed-step marcher with empty-space
// skipping (NA/nerfacc/cuda/csrc/ray_marching.cu:9-192,
// NA/nerfacc/cuda/csrc/include/helpers_contraction.h:16-114) so that, for
// the same rays, t_min, step size and grid, the emitted samples are
// bit-identical: every floating-point operation below is written with an
// explicit rounding intrinsic in the order the reference evaluates it.
// nvcc contracts the reference's `origin + t_mid * dir` into one FMA
// (default -fmad=true); all other products there are exact scalings by 0.5
// or are not followed by an addition, so they are plain roundings.
#include "common.cuh"
#include "scan.cuh"

#include <string.h>

#include <mutex>

namespace sn {

static thread_local char g_err[512];
static unsigned long long g_launches = 0;

void count_launches(int k) { __atomic_fetch_add(&g_launches, (unsigned long long)k, __ATOMIC_RELAXED); }

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

int num_sms() {
  static int cached = 0;
  if (cached == 0) {
    int dev = 0, v = 0;
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && v > 0)
      cached = v;
    else
      cached = 132;
  }
  return cached;
}

// Scans each tile, adds the tile offset and writes packed_info = {offset, count}.
__global__ void __launch_bounds__(kScanThreads)
scan_tile_apply(const int32_t* __restrict__ in, int64_t n, const int32_t* __restrict__ tile_offsets,
                int32_t* __restrict__ packed, int32_t* __restrict__ total,
                const int32_t* __restrict__ live = nullptr) {
  chained();
  if (live) n = min(n, (int64_t)*live);   // entries at or past *live are neither read nor written
  if ((int64_t)blockIdx.x * kScanTile >= n) {
    if (!tile_offsets && threadIdx.x == 0 && total) *total = 0;
    return;
  }
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int v[kScanItems], c[kScanItems];
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) c[i] = v[i] = (base + i < n) ? in[base + i] : 0;
  int tot = block_exclusive_scan(v);
  const int off = tile_offsets ? tile_offsets[blockIdx.x] : 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    if (base + i < n) {
      int2 pk = make_int2(v[i] + off, c[i]);
      reinterpret_cast<int2*>(packed)[base + i] = pk;
    }
  }
  if (!tile_offsets && threadIdx.x == 0 && total) *total = tot;
}

int pack_counts(int64_t n, const int32_t* counts, int32_t* packed, int32_t* total, void* ws,
                cudaStream_t st, const int32_t* live = nullptr) {
  if (n == 0) {
    if (total) {
      if (cudaMemsetAsync(total, 0, sizeof(int32_t), st) != cudaSuccess) {
        set_error("pack_counts: memset failed");
        return SN_ERR_CUDA;
      }
    }
    return SN_OK;
  }
  const int64_t n_tiles = (n + kScanTile - 1) / kScanTile;
  if (n_tiles == 1) {
    launch_chained(scan_tile_apply, 1, kScanThreads, 0, st, counts, n, nullptr, packed, total, live);
    return check_launch("pack_counts");
  }
  SN_REQUIRE(ws != nullptr, "pack_counts: workspace required for n=%lld", (long long)n);
  int32_t* tiles = reinterpret_cast<int32_t*>(ws);
  scan_tile_reduce<<<(unsigned)n_tiles, kScanThreads, 0, st>>>(counts, n, tiles, live);
  scan_tile_offsets<<<1, kScanThreads, 0, st>>>(tiles, n_tiles, total, live, n);
  scan_tile_apply<<<(unsigned)n_tiles, kScanThreads, 0, st>>>(counts, n, tiles, packed, nullptr, live);
  return check_launch("pack_counts", 3);
}

struct SmemLimit {
  int dev;
  const void* fn;
  size_t bytes;
};
static std::mutex g_smem_mu;
static SmemLimit g_smem_set[64];
static int g_smem_n = 0;

int ensure_smem_limit(const void* fn, size_t bytes, const char* what) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    set_error("%s: cudaGetDevice failed: %s", what, cudaGetErrorString(e));
    return SN_ERR_CUDA;
  }
  std::lock_guard<std::mutex> lock(g_smem_mu);
  for (int i = 0; i < g_smem_n; ++i)
    if (g_smem_set[i].dev == dev && g_smem_set[i].fn == fn && g_smem_set[i].bytes >= bytes) return SN_OK;
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) {
    set_error("%s: cannot set the shared memory limit to %zu bytes: %s", what, bytes, cudaGetErrorString(e));
    return SN_ERR_CUDA;
  }
  if (g_smem_n < 64) g_smem_set[g_smem_n++] = SmemLimit{dev, fn, bytes};
  return SN_OK;
}

// Static scratch of sn_pack_counts_static: tile sums of up to kPackStaticMaxTiles
// tiles.  Its device address is looked up once per device (with that device
// current) and cached for the life of the process.  cudaDeviceReset destroys
// the module that holds the array, and a later call would write through the
// stale address, so a process that resets a device must not call the entry
// point on that device again.
constexpr int64_t kPackStaticMaxTiles = 4096;
constexpr int64_t kPackStaticMaxEntries = kPackStaticMaxTiles * kScanTile;
static __device__ __align__(256) int32_t g_pack_scratch[kPackStaticMaxTiles];
constexpr int kPackScratchDevices = 64;
static std::mutex g_pack_scratch_mu;
static int32_t* g_pack_scratch_ptr[kPackScratchDevices];

int pack_scratch_for_current_device(int32_t** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    set_error("pack_counts_static: cudaGetDevice failed: %s", cudaGetErrorString(e));
    return SN_ERR_CUDA;
  }
  SN_REQUIRE(dev >= 0 && dev < kPackScratchDevices, "pack_counts_static: device %d out of range", dev);
  std::lock_guard<std::mutex> lock(g_pack_scratch_mu);
  if (!g_pack_scratch_ptr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_pack_scratch);
    if (e != cudaSuccess || p == nullptr) {
      set_error("pack_counts_static: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
      return SN_ERR_CUDA;
    }
    g_pack_scratch_ptr[dev] = static_cast<int32_t*>(p);
  }
  *out = g_pack_scratch_ptr[dev];
  return SN_OK;
}

// ---------------------------------------------------------------------------
// counts / unpack
// ---------------------------------------------------------------------------
__global__ void count_indices_kernel(int64_t n, const int64_t* __restrict__ idx, int64_t n_rays,
                                     int32_t* __restrict__ counts) {
  // warp-uniform loop so the whole warp takes part in every ballot/match
  const int lane = threadIdx.x & 31;
  const int64_t warp0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) - lane;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t b = warp0; b < n; b += stride) {
    const int64_t s = b + lane;
    const int64_t r = s < n ? idx[s] : -1;
    const bool ok = r >= 0 && r < n_rays;
    const unsigned m = __ballot_sync(0xffffffffu, ok);
    if (ok) {
      // samples of one ray are usually adjacent: one atomic per distinct key
      const unsigned peers = __match_any_sync(m, r);
      if (lane == __ffs(peers) - 1) atomicAdd(&counts[r], __popc(peers));
    }
  }
}

__global__ void unpack_info_kernel(int64_t n_rays, const int32_t* __restrict__ packed,
                                   int64_t n_samples, int64_t* __restrict__ out) {
  // one warp per ray: lanes write the ray's samples cooperatively
  const int lane = threadIdx.x & 31;
  for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; r < n_rays;
       r += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const int base = packed[2 * r], cnt = packed[2 * r + 1];
    for (int j = lane; j < cnt; j += 32) {
      int64_t s = (int64_t)base + j;
      if (s < n_samples) out[s] = r;
    }
  }
}

// ---------------------------------------------------------------------------
// marcher
// ---------------------------------------------------------------------------
struct GridView {
  const float* roi;  // device, 6 floats: {min xyz, max xyz}
  float lo[3], hi[3];
  int res[3];
  const uint8_t* bits;
  int ctype;
  float ext[3], rext[3], rres[3];  // extent; exact reciprocals of extent and resolution, or 0
  float scale[3], rscale[3];       // resolution / extent and its reciprocal, where both are exact
};

// 1/v when v is a normal power of two (then x * (1/v) rounds exactly as x / v,
// both being the correctly rounded value of the same real number), else 0.
__device__ __forceinline__ float pow2_recip(float v) {
  const uint32_t b = __float_as_uint(v);
  const uint32_t e = (b >> 23) & 0xFFu;
  const bool p2 = (b & 0x807FFFFFu) == 0u && e >= 1u && e <= 253u;
  return p2 ? __uint_as_float((254u - e) << 23) : 0.0f;
}
// x / v, as a multiplication when r = pow2_recip(v) is nonzero (same bits).
__device__ __forceinline__ float div_by(float x, float v, float r) {
  return r != 0.0f ? __fmul_rn(x, r) : __fdiv_rn(x, v);
}

__device__ __forceinline__ void load_roi(GridView& g) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    g.lo[d] = g.roi[d];
    g.hi[d] = g.roi[3 + d];
    g.ext[d] = __fsub_rn(g.hi[d], g.lo[d]);
    g.rext[d] = pow2_recip(g.ext[d]);
    g.rres[d] = pow2_recip((float)g.res[d]);
    g.scale[d] = g.rext[d] * (float)g.res[d];
    g.rscale[d] = g.rres[d] * g.ext[d];
  }
}

// roi -> [0,1]^3 and the two unbounded contractions
// (NA/nerfacc/cuda/csrc/include/helpers_contraction.h:16-114).
__device__ __forceinline__ void contract(const GridView& g, const float p[3], float u[3]) {
#pragma unroll
  for (int d = 0; d < 3; ++d) u[d] = div_by(__fsub_rn(p[d], g.lo[d]), g.ext[d], g.rext[d]);
  if (g.ctype == SN_CONTRACTION_UN_BOUNDED_TANH) {
#pragma unroll
    for (int d = 0; d < 3; ++d) u[d] = __fmaf_rn(tanhf(__fsub_rn(u[d], 0.5f)), 0.5f, 0.5f);
  } else if (g.ctype == SN_CONTRACTION_UN_BOUNDED_SPHERE) {
#pragma unroll
    for (int d = 0; d < 3; ++d) u[d] = __fmaf_rn(u[d], 2.0f, -1.0f);
    float nsq = __fmaf_rn(u[2], u[2], __fmaf_rn(u[1], u[1], __fmul_rn(u[0], u[0])));
    float nrm = sqrtf(nsq);
    if (nrm > 1.0f) {
      float k = __fsub_rn(2.0f, __fdiv_rn(1.0f, nrm));
#pragma unroll
      for (int d = 0; d < 3; ++d) u[d] = __fmul_rn(k, __fdiv_rn(u[d], nrm));
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) u[d] = __fmaf_rn(u[d], 0.25f, 0.5f);
  }
}

// grid_occupied_at + grid_idx_at (NA/nerfacc/cuda/csrc/ray_marching.cu:16-45):
// AABB rejection, contraction, truncating int conversion, clamp, x-major index.
__device__ __forceinline__ bool occupied_at(const GridView& g, const float p[3]) {
  if (g.ctype == SN_CONTRACTION_AABB &&
      (p[0] < g.lo[0] || p[0] > g.hi[0] || p[1] < g.lo[1] || p[1] > g.hi[1] ||
       p[2] < g.lo[2] || p[2] > g.hi[2]))
    return false;
  float u[3];
  contract(g, p, u);
  int ix[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    int v = (int)__fmul_rn(u[d], (float)g.res[d]);
    v = v < 0 ? 0 : v;
    v = v > g.res[d] - 1 ? g.res[d] - 1 : v;
    ix[d] = v;
  }
  const int idx = ix[0] * (g.res[1] * g.res[2]) + ix[1] * g.res[2] + ix[2];
  return __ldg(g.bits + idx) != 0;
}

// Grid coordinates of a point: the contraction of an AABB grid times the
// resolution, whose truncation is grid_idx_at's cell.  P2: extents and
// resolutions are powers of two (every division is exact scaling, so the two
// factors of an axis are one multiplication with the same bits).
template <bool P2>
__device__ __forceinline__ void grid_coords(const GridView& g, const float p[3], float xu[3]) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float x = __fsub_rn(p[d], g.lo[d]);
    xu[d] = P2 ? __fmul_rn(x, g.scale[d]) : __fmul_rn(div_by(x, g.ext[d], g.rext[d]), (float)g.res[d]);
  }
}

// occupied_at of an AABB grid from its grid coordinates.
__device__ __forceinline__ bool occupied_at_coords(const GridView& g, const float p[3], const float xu[3]) {
  if (p[0] < g.lo[0] || p[0] > g.hi[0] || p[1] < g.lo[1] || p[1] > g.hi[1] || p[2] < g.lo[2] || p[2] > g.hi[2])
    return false;
  int ix[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) ix[d] = min((int)xu[d], g.res[d] - 1);
  return __ldg(g.bits + ((ix[0] * g.res[1] + ix[1]) * g.res[2] + ix[2])) != 0;
}

// distance_to_next_voxel + the target of advance_to_next_voxel
// (NA/nerfacc/cuda/csrc/ray_marching.cu:47-75): the ray parameter that the
// marcher steps to from an empty cell, in dt_min increments (at least one) so
// samples stay on the marching lattice.
template <bool P2>
__device__ __forceinline__ float skip_target(const GridView& g, float t, const float xu[3], const float dir[3],
                                             const float inv[3], float far) {
  float tx[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float f = floorf(__fadd_rn(__fadd_rn(xu[d], 0.5f), copysignf(0.5f, dir[d])));
    const float x = __fmul_rn(__fsub_rn(f, xu[d]), inv[d]);
    tx[d] = P2 ? __fmul_rn(x, g.rscale[d]) : __fmul_rn(div_by(x, (float)g.res[d], g.rres[d]), g.ext[d]);
  }
  float dist = fminf(fminf(tx[0], tx[1]), tx[2]);
  dist = fmaxf(dist, 0.0f);
  return fminf(__fadd_rn(t, dist), far);
}

__device__ __forceinline__ float step_to(float t, float target, float dt_min) {
  do {
    t = __fadd_rn(t, dt_min);
  } while (t < target);
  return t;
}

__device__ __forceinline__ float calc_dt(float t, float cone, float dt_min, float dt_max) {
  return fminf(fmaxf(__fmul_rn(t, cone), dt_min), dt_max);
}

struct MarchArgs {
  int64_t n_rays;
  const float* rays_o;
  const float* rays_d;
  const float* t_min;
  const float* t_max;
  const float* jitter;
  GridView grid;
  float step;
  const float* step_dev;  // nullable: the step size in device memory (overrides step)
  float cone;
  int64_t max_iters;
  const int32_t* packed;
  int64_t capacity;
  int32_t* num_steps;
  int64_t* ray_indices;
  float* t_starts;
  float* t_ends;
  int32_t* status;
  float4* runs;           // nullable: kMarchRuns per ray, see sn_march_runs
  const uint32_t* blocks;  // nullable: occupied blocks of the grid, see march_blocks_kernel
  int32_t* packed_out;     // march_expand_kernel from counts: packed_info and the total, written
  int32_t* total;
};

// The reference marcher (NA/nerfacc/cuda/csrc/ray_marching.cu:135-185) walks one ray sequentially:
//   while t_mid < far: if occupied(origin + t_mid*dir): emit [t0, t1], t0 = t1,
//   t1 = t0 + dt, t_mid = (t0 + t1)/2; else t_mid = DDA skip, t0/t1 = t_mid -/+ dt/2.
// The marcher below gives the same samples bit for bit.
//
// Consecutive occupied steps form a run: every sample of a run follows from
// its first state (t0, t1) by additions alone.  A counting march keeps the runs
// (at most kMarchRuns a ray), and the samples are then written from them
// without a second march.
constexpr int kMarchRuns = 16;

struct MarchRay {
  float o[3], d[3], inv[3];
  float far, dt_min, cone;
};
constexpr float kMarchDtMax = 1e10f;

// cone_angle == 0: calc_dt(t) = clamp(t * 0, dt_min, dt_max) is dt_min for every t.
template <bool CONE>
__device__ __forceinline__ float step_dt(const MarchRay& r, float t) {
  return CONE ? calc_dt(t, r.cone, r.dt_min, kMarchDtMax) : r.dt_min;
}

// Loads ray `ray` and its first state.
template <bool CONE>
__device__ __forceinline__ void load_ray(const MarchArgs& a, int64_t ray, MarchRay& r, float& t0, float& t1,
                                         float& tm) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    r.o[k] = a.rays_o[3 * ray + k];
    r.d[k] = a.rays_d[3 * ray + k];
    r.inv[k] = __fdiv_rn(1.0f, r.d[k]);
  }
  r.dt_min = a.step_dev ? *a.step_dev : a.step;
  r.cone = a.cone;
  r.far = a.t_max[ray];
  t0 = a.t_min[ray];
  if (a.jitter) t0 = __fadd_rn(t0, __fmul_rn(a.jitter[ray], r.dt_min));
  t1 = __fadd_rn(t0, step_dt<CONE>(r, t0));
  tm = __fmul_rn(__fadd_rn(t0, t1), 0.5f);
}

__device__ __forceinline__ void ray_at(const MarchRay& r, float t, float p[3]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) p[k] = __fmaf_rn(t, r.d[k], r.o[k]);
}

// State around an occupied position that a skip reached.
template <bool CONE>
__device__ __forceinline__ void state_at(const MarchRay& r, float tm, float& t0, float& t1) {
  const float h = __fmul_rn(step_dt<CONE>(r, tm), 0.5f);
  t0 = __fsub_rn(tm, h);
  t1 = __fadd_rn(tm, h);
}

// ---- occupied blocks -----------------------------------------------------------
// The grid in at most 32 blocks per axis, one bit per block that holds an
// occupied cell (bit = z, 4 KB in all).  A point whose block and 26 neighbours
// are empty certifies a stretch of the ray around it, so 32 lanes tell in
// one round where the last occupied cell on the ray can be; behind it the
// marcher emits nothing, whatever positions it would visit.
constexpr int kBlockAxis = 32;
// Rays from which on the blocks pay for their kernel (counting with / without
// them at a step of 2/1024: 2,048 rays 36 / 29 us, 8,192 53 / 51, 32,768 115 /
// 150, 313,344 0.69 / 1.04 ms).
constexpr int64_t kBlockRays = 16384;
struct BlockDims {
  int e[3];  // cells per block edge
};
static inline BlockDims block_dims(const GridView& g) {
  BlockDims b;
  for (int d = 0; d < 3; ++d) b.e[d] = (g.res[d] + kBlockAxis - 1) / kBlockAxis;
  return b;
}
__device__ __forceinline__ int block_edge(int res) { return (res + kBlockAxis - 1) / kBlockAxis; }

// One warp per (x, y) column of blocks, lane = z.  Blocks that are whole aligned
// words along z (the 128^3 grid's) are read as words, coalesced over the warp.
__global__ void __launch_bounds__(256)
march_blocks_kernel(const uint8_t* __restrict__ bits, int rx, int ry, int rz, BlockDims b, uint32_t* __restrict__ out) {
  const int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), z = threadIdx.x & 31;
  const int x0 = (w / kBlockAxis) * b.e[0], y0 = (w % kBlockAxis) * b.e[1], z0 = z * b.e[2];
  const int x1 = min(x0 + b.e[0], rx), y1 = min(y0 + b.e[1], ry), z1 = min(z0 + b.e[2], rz);
  const bool words = b.e[2] == 4 && (rz & 3) == 0 && (reinterpret_cast<uintptr_t>(bits) & 3) == 0;
  uint32_t any = 0;
  for (int x = x0; x < x1; ++x) {
    const uint8_t* row = bits + ((int64_t)x * ry + y0) * rz + z0;
    if (words) {
      if (z0 < rz) {
#pragma unroll 4
        for (int y = y0; y < y1; ++y, row += rz) any |= __ldg(reinterpret_cast<const uint32_t*>(row));
      }
    } else {
      for (int y = y0; y < y1; ++y, row += rz)
        for (int k = 0; k < z1 - z0; ++k) any |= row[k];
    }
  }
  const uint32_t word = __ballot_sync(0xffffffffu, any != 0);
  if (z == 0) out[w] = word;
}

// Ray parameter past which no position of the ray from t on is occupied (far
// where that is not known).  Lane l looks at the middle of the l-th stretch,
// whose half length moves the ray by less than a block edge along every axis:
// every cell of the stretch then lies in the point's block or one beside it.
// The hundredth of a cell that is left covers the rounding.  In cells: a position, its
// difference from the box's side and the two factors after it are at most 2^-22 (|p| +
// the box's largest coordinate) off, 0.001 at the limit of 4,096 for the tested point
// and 0.002 for the others, at most twice as far out; the tested point's parameter is
// two roundings off, 2 x 2^-24 |t|, 0.0048 at 40,000.  Beyond these limits the stretch
// counts as occupied.  A block index past the grid is clamped: the blocks beside it
// are then among those that are tested.
__device__ __forceinline__ float last_occupied(const GridView& g, const uint32_t* __restrict__ blocks,
                                               const MarchRay& r, float t, int lane) {
  float rate[3], cells[3], half = 1e30f, fastest = 0.0f, reach = 0.0f;
  int e[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    e[d] = block_edge(g.res[d]);
    cells[d] = (float)g.res[d] / g.ext[d];     // per unit of length
    rate[d] = fabsf(r.d[d]) * cells[d];        // per unit of t
    half = fminf(half, ((float)e[d] - 0.01f) / rate[d]);
    fastest = fmaxf(fastest, rate[d]);
    reach = fmaxf(reach, fmaxf(fabsf(g.lo[d]), fabsf(g.hi[d])));
  }
  half *= 0.9999f;
  const float c = t + (float)(2 * lane + 1) * half;
  float p[3], xu[3];
  ray_at(r, c, p);
  grid_coords<false>(g, p, xu);
  bool sure = fabsf(c) * fastest < 40000.0f;
  int b[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    sure = sure && (fabsf(p[d]) + reach) * cells[d] <= 4096.0f;
    const int nb = (g.res[d] + e[d] - 1) / e[d];
    b[d] = min(max((int)floorf(xu[d] / (float)e[d]), 0), nb - 1);
  }
  uint32_t any = 0;
#pragma unroll
  for (int dx = -1; dx <= 1; ++dx)
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy) {
      const int bx = b[0] + dx, by = b[1] + dy;
      if (bx >= 0 && bx < kBlockAxis && by >= 0 && by < kBlockAxis) any |= __ldg(blocks + bx * kBlockAxis + by);
    }
  const uint32_t near_z = b[2] > 0 ? 7u << (b[2] - 1) : 3u;
  const bool before_far = t + (float)(2 * lane) * half < r.far;
  const uint32_t open = __ballot_sync(0xffffffffu, before_far && (!sure || (any & near_z)));
  if (!(t + 64.0f * half >= r.far) || (open >> 31)) return r.far;   // the stretches end before the ray does
  return open ? fminf(r.far, t + (float)(2 * (32 - __clz(open)) + 1) * half) : t;
}

// ---- warp per ray ------------------------------------------------------------
// The warp looks at 64 consecutive positions at a time, two per lane (position
// lane + 32 i), so a ray costs one grid round trip per 64 steps:
//  * In a run, position k's state is the one after k occupied steps; a ballot
//    finds the first that is empty or past far.  Those before it are samples.
//  * In empty space, position k is k additions of dt_min past the first.  The
//    sequential marcher visits some of them: a skip from an empty position goes
//    to the first position at or past its target.  The guess is that it
//    visits the first position of every cell; each lane checks its own
//    guess with its own target, and where all agree up to the first guessed
//    position that is occupied or past far, that is where the marcher
//    stops (induction from the first, which is visited).  Where one does not
//    (a position within rounding of a cell's side), the walk goes on from the
//    last confirmed position by its own target.
// With a constant step the k-th addition is guessed in closed form
// (s + k delta, one rounding) and accepted when every lane's own step agrees with
// the sequential rule; otherwise (a binade crossing that rounds, a tie, cone
// > 0) the additions are replayed one by one.
// Bound by instruction issue for many rays and by the chain of round trips for
// few.  Measured (samples identical) on a grid like a trained one, step 2/1024,
// against 8 lanes each chaining skips of its own: counting 2,048 rays 73 -> 29
// us, 313,344 rays 2.31 -> 0.69 ms; the samples, formerly a second march of
// 2.48 ms, are written from the runs in 0.12 ms (4.5 TB/s).
constexpr int kPos = 2;           // positions per lane
constexpr int kWindow = 32 * kPos;

__device__ __forceinline__ float at64(const float v[kPos], int k) {
  const float x = __shfl_sync(0xffffffffu, v[0], k & 31), y = __shfl_sync(0xffffffffu, v[1], k & 31);
  return k < 32 ? x : y;
}
__device__ __forceinline__ uint64_t ballot64(bool b0, bool b1) {
  return (uint64_t)__ballot_sync(0xffffffffu, b0) | (uint64_t)__ballot_sync(0xffffffffu, b1) << 32;
}

// States after k occupied steps from (t0, t1), k = lane + 32 i.
template <bool CONE>
__device__ __forceinline__ void run_states(const MarchRay& r, float t0, float t1, int lane, float l0[kPos],
                                           float l1[kPos]) {
  bool exact = false;
  if (!CONE) {
    const float delta = __fsub_rn(__fadd_rn(t1, r.dt_min), t1);
    bool ok = true;
#pragma unroll
    for (int i = 0; i < kPos; ++i) {
      const int k = lane + 32 * i;
      l0[i] = k > 0 ? __fmaf_rn((float)(k - 1), delta, t1) : t0;
      l1[i] = k > 0 ? __fmaf_rn((float)k, delta, t1) : t1;
      ok = ok && (k == 0 || __fadd_rn(l0[i], r.dt_min) == l1[i]);
    }
    exact = __all_sync(0xffffffffu, ok);
  }
  if (!exact) {
    float a0 = t0, a1 = t1;
#pragma unroll
    for (int i = 0; i < kPos; ++i) {
      for (int s = 0; s < (i == 0 ? lane : 32); ++s) {
        a0 = a1;
        a1 = __fadd_rn(a0, step_dt<CONE>(r, a0));
      }
      l0[i] = a0;
      l1[i] = a1;
    }
  }
}

// Walks empty space from the visited position s (not tested yet).  Returns true
// with s at the next occupied position; false where there is none before end
// (far, or where last_occupied allows none) or past the limit.
template <bool P2>
__device__ __forceinline__ bool walk_empty(const GridView& g, const MarchRay& r, int lane, float end,
                                           float& s, int64_t& iters, int64_t max_iters, bool& limit) {
  while (true) {
    float sk[kPos], T[kPos];
    {
      const float delta = __fsub_rn(__fadd_rn(s, r.dt_min), s);
      bool ok = true;
#pragma unroll
      for (int i = 0; i < kPos; ++i) {
        const int k = lane + 32 * i;
        sk[i] = k > 0 ? __fmaf_rn((float)k, delta, s) : s;
        ok = ok && (k == 0 || __fadd_rn(k > 1 ? __fmaf_rn((float)(k - 1), delta, s) : s, r.dt_min) == sk[i]);
      }
      if (!__all_sync(0xffffffffu, ok)) {
        float a = s;
#pragma unroll
        for (int i = 0; i < kPos; ++i) {
          for (int q = 0; q < (i == 0 ? lane : 32); ++q) a = __fadd_rn(a, r.dt_min);
          sk[i] = a;
        }
      }
    }
    bool first[kPos], stop[kPos];
    uint32_t key[kPos];
#pragma unroll
    for (int i = 0; i < kPos; ++i) {
      float p[3], xu[3];
      ray_at(r, sk[i], p);
      grid_coords<P2>(g, p, xu);
      const bool in = sk[i] < end;
      const bool occ = in && occupied_at_coords(g, p, xu);
      T[i] = skip_target<P2>(g, sk[i], xu, r.d, r.inv, r.far);
      // tells neighbouring cells apart; a collision only costs a failed check
      key[i] = (uint32_t)(int)floorf(xu[0]) + ((uint32_t)(int)floorf(xu[1]) << 10) +
               ((uint32_t)(int)floorf(xu[2]) << 20);
      stop[i] = occ || !in;
      first[i] = !in;
    }
    uint32_t before = 0;
#pragma unroll
    for (int i = 0; i < kPos; ++i) {
      const uint32_t up = __shfl_up_sync(0xffffffffu, key[i], 1);
      first[i] = first[i] || key[i] != (lane > 0 ? up : before) || (lane == 0 && i == 0);
      before = __shfl_sync(0xffffffffu, key[i], 31);
    }
    const uint64_t N = ballot64(first[0], first[1]);
    const uint64_t S = N & ballot64(stop[0], stop[1]);
    bool wrong[kPos];
#pragma unroll
    for (int i = 0; i < kPos; ++i) {
      const int k = lane + 32 * i;
      const uint64_t rest = k < kWindow - 1 ? N >> (k + 1) : 0ull;
      const int b = rest ? k + __ffsll((long long)rest) : k;
      const float sb = at64(sk, b), sp = at64(sk, b > 0 ? b - 1 : 0);
      wrong[i] = first[i] && rest && !(sb >= T[i] && (b - 1 == k || sp < T[i]));
    }
    const uint64_t bad = ballot64(wrong[0], wrong[1]);
    const int k = S ? __ffsll((long long)S) - 1 : kWindow;
    if (k < kWindow && !(bad & ((1ull << k) - 1ull))) {
      iters += __popcll(N & ((1ull << k) - 1ull));
      s = at64(sk, k);
      return s < end;
    }
    // on from the last confirmed position, which is empty
    const int e = bad ? __ffsll((long long)bad) - 1 : 63 - __clzll((long long)N);
    iters += __popcll(N & (~0ull >> (63 - e)));
    s = step_to(at64(sk, e), at64(T, e), r.dt_min);
    if (!(s < end)) return false;
    if (iters > max_iters) {
      limit = true;
      return false;
    }
  }
}

// Marches one ray with the whole warp.  FILL: samples to [base, base + room)
// below the capacity.  Returns the number of samples.  P2: an AABB grid whose
// extents and resolutions are powers of two (SuperNormal's is), which leaves
// out the divisions and the contractions: half the instructions, and code that
// stays in the instruction cache.
template <bool FILL, bool CONE, bool P2>
__device__ __forceinline__ int64_t march_ray_in(const MarchArgs& a, const GridView& g, int64_t ray, int64_t base,
                                             int64_t room, int lane) {
  MarchRay r;
  float t0, t1, tm0;
  load_ray<CONE>(a, ray, r, t0, t1, tm0);
  const bool aabb = P2 || g.ctype == SN_CONTRACTION_AABB;
  float end = r.far;
  int64_t j = 0, iters = 0;
  bool overflow = false, limit = false;
  float run_t0 = 0.0f, run_t1 = 0.0f;
  int run_len = 0, n_runs = 0;
  bool more = true;
  if (aabb) {  // rays usually start in empty space
    const float tm = tm0;
    // worth a round only where the walk could take several
    if (a.blocks && r.far - tm0 > 2 * kWindow * r.dt_min) end = last_occupied(g, a.blocks, r, tm0, lane);
    more = tm0 < end && walk_empty<P2>(g, r, lane, end, tm0, iters, a.max_iters, limit);
    if (more && tm0 != tm) state_at<CONE>(r, tm0, t0, t1);
  }
  while (more) {
    float l0[kPos], l1[kPos], tm[kPos];
    run_states<CONE>(r, t0, t1, lane, l0, l1);
    bool inside[kPos], empty[kPos];
#pragma unroll
    for (int i = 0; i < kPos; ++i) {
      // the first position of a state that a skip reached is the skip's own result
      tm[i] = lane + 32 * i == 0 ? tm0 : __fmul_rn(__fadd_rn(l0[i], l1[i]), 0.5f);
      float p[3];
      ray_at(r, tm[i], p);
      inside[i] = tm[i] < r.far;
      bool occ;
      if (P2) {
        float xu[3];
        grid_coords<true>(g, p, xu);
        occ = inside[i] && occupied_at_coords(g, p, xu);
      } else {
        occ = inside[i] && occupied_at(g, p);
      }
      empty[i] = !occ;
    }
    const uint64_t em = ballot64(empty[0], empty[1]);
    const uint64_t im = ballot64(inside[0], inside[1]);
    int m = em ? __ffsll((long long)em) - 1 : kWindow;  // occupied run length
    if (iters + m > a.max_iters) {
      m = (int)max(a.max_iters - iters, (int64_t)0);
      limit = true;
    }
    if (FILL) {
#pragma unroll
      for (int i = 0; i < kPos; ++i) {
        const int k = lane + 32 * i;
        if (k < m) {
          const int64_t jj = j + k;
          if (jj < room && base + jj < a.capacity) {
            a.t_starts[base + jj] = l0[i];
            a.t_ends[base + jj] = l1[i];
            a.ray_indices[base + jj] = ray;
          } else {
            overflow = true;
          }
        }
      }
    } else if (m > 0) {
      if (run_len == 0) {
        run_t0 = t0;
        run_t1 = t1;
      }
      run_len += m;
    }
    j += m;
    iters += m + 1;
    if (limit) break;
    if (m == kWindow) {  // all occupied: on after the last
      t0 = at64(l1, kWindow - 1);
      t1 = __fadd_rn(t0, step_dt<CONE>(r, t0));
      tm0 = __fmul_rn(__fadd_rn(t0, t1), 0.5f);
      continue;
    }
    if (!FILL && run_len > 0) {
      if (a.runs && lane == 0 && n_runs < kMarchRuns)
        a.runs[ray * kMarchRuns + n_runs] = make_float4(run_t0, run_t1, __int_as_float(run_len), 0.0f);
      ++n_runs;
      run_len = 0;
    }
    // position m holds the sequential state at the first that is not occupied
    if (!((im >> m) & 1ull)) break;
    if (aabb) {
      tm0 = at64(tm, m);
      more = tm0 < end && walk_empty<P2>(g, r, lane, end, tm0, iters, a.max_iters, limit);
      if (more) state_at<CONE>(r, tm0, t0, t1);
    } else {
      t0 = at64(l1, m);
      t1 = __fadd_rn(t0, step_dt<CONE>(r, t0));
      tm0 = __fmul_rn(__fadd_rn(t0, t1), 0.5f);
      more = tm0 < r.far;
    }
    if (iters > a.max_iters) {
      limit = true;
      break;
    }
  }
  if (!FILL && run_len > 0) {  // the limit struck inside a run
    if (a.runs && lane == 0 && n_runs < kMarchRuns)
      a.runs[ray * kMarchRuns + n_runs] = make_float4(run_t0, run_t1, __int_as_float(run_len), 0.0f);
    ++n_runs;
  }
  if (lane == 0) {
    if (!FILL && a.runs && n_runs > 0) a.runs[ray * kMarchRuns].w = __int_as_float(n_runs);
    if (limit) atomicOr(a.status, SN_STATUS_MARCH_LIMIT);
  }
  if (FILL && __any_sync(0xffffffffu, overflow) && lane == 0) atomicOr(a.status, SN_STATUS_CAPACITY);
  return j;
}

template <bool FILL, bool CONE>
__device__ __forceinline__ int64_t march_ray(const MarchArgs& a, const GridView& g, int64_t ray, int64_t base,
                                             int64_t room, int lane) {
  bool p2 = g.ctype == SN_CONTRACTION_AABB;
#pragma unroll
  for (int d = 0; d < 3; ++d) p2 = p2 && g.rext[d] != 0.0f && g.rres[d] != 0.0f;
  return p2 ? march_ray_in<FILL, CONE, true>(a, g, ray, base, room, lane)
            : march_ray_in<FILL, CONE, false>(a, g, ray, base, room, lane);
}

// Modes: count (num_steps and runs), fill at packed_info offsets, or fill into
// fixed slots ray*slot_stride (padded; num_steps written too).
template <int MODE, bool CONE>  // MODE: 0 count, 1 fill packed, 2 fill padded
__global__ void __launch_bounds__(128) march_warp_kernel(MarchArgs a, int64_t slot_stride) {
  chained();
  const int lane = threadIdx.x & 31;
  const int64_t ray = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  if (ray >= a.n_rays) return;  // whole warp exits together
  GridView g = a.grid;
  load_roi(g);
  int64_t base = 0, room = 0;
  if (MODE == 1) {
    base = a.packed[2 * ray];
    room = a.packed[2 * ray + 1];
  } else if (MODE == 2) {
    base = ray * slot_stride;
    room = slot_stride;
  }
  const int64_t j = march_ray<MODE != 0, CONE>(a, g, ray, base, room, lane);
  if (MODE != 1 && lane == 0) a.num_steps[ray] = (int32_t)j;
  if (MODE == 0 && lane == 0 && slot_stride > 0 && j > slot_stride) atomicOr(a.status, SN_STATUS_CAPACITY);
}

// Samples of the recorded runs at the packed_info offsets, one warp per ray;
// a ray with more runs than were kept is marched again.  COUNTS: the offsets are
// formed here, from num_steps.
template <bool CONE, bool COUNTS>
__global__ void __launch_bounds__(128, 12) march_expand_kernel(MarchArgs a) {
  chained();
  const int lane = threadIdx.x & 31;
  const int64_t ray = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  int64_t base;
  int room;
  if constexpr (COUNTS) {
    const int2 pk = packed_from_counts(a.num_steps, a.n_rays, a.packed_out, a.total);
    base = pk.x;
    room = pk.y;
  } else {
    if (ray >= a.n_rays) return;
    base = a.packed[2 * ray];
    room = a.packed[2 * ray + 1];
  }
  if (room <= 0) return;
  // most rays have few runs: half of the ray's slots first
  float4 mine = a.runs[ray * kMarchRuns + (lane & (kMarchRuns / 2 - 1))];
  const int n_runs = __float_as_int(__shfl_sync(0xffffffffu, mine.w, 0));
  if (n_runs > kMarchRuns) {
    GridView g = a.grid;
    load_roi(g);
    march_ray<true, CONE>(a, g, ray, base, room, lane);
    return;
  }
  if (n_runs > kMarchRuns / 2) mine = a.runs[ray * kMarchRuns + (lane & (kMarchRuns - 1))];
  MarchRay r;
  r.dt_min = a.step_dev ? *a.step_dev : a.step;
  r.cone = a.cone;
  int64_t j = 0;
  bool overflow = false;
  for (int q = 0; q < n_runs; ++q) {
    float t0 = __shfl_sync(0xffffffffu, mine.x, q), t1 = __shfl_sync(0xffffffffu, mine.y, q);
    const int len = __float_as_int(__shfl_sync(0xffffffffu, mine.z, q));
    for (int k0 = 0; k0 < len; k0 += kWindow) {
      float l0[kPos], l1[kPos];
      run_states<CONE>(r, t0, t1, lane, l0, l1);
#pragma unroll
      for (int i = 0; i < kPos; ++i) {
        const int k = k0 + lane + 32 * i;
        if (k < len) {
          const int64_t o = base + j + k;
          if (o < a.capacity) {
            a.t_starts[o] = l0[i];
            a.t_ends[o] = l1[i];
            a.ray_indices[o] = ray;
          } else {
            overflow = true;
          }
        }
      }
      if (k0 + kWindow < len) {
        t0 = at64(l1, kWindow - 1);
        t1 = __fadd_rn(t0, step_dt<CONE>(r, t0));
      }
    }
    j += len;
  }
  if (__any_sync(0xffffffffu, overflow) && lane == 0) atomicOr(a.status, SN_STATUS_CAPACITY);
}

// Copy padded per-ray samples (ray*stride + j, j < count) to packed offsets.
__global__ void compact_padded_kernel(int64_t n_rays, int64_t stride, const int32_t* __restrict__ packed,
                                      const int64_t* __restrict__ ri_in, const float* __restrict__ ts_in,
                                      const float* __restrict__ te_in, int64_t* __restrict__ ri_out,
                                      float* __restrict__ ts_out, float* __restrict__ te_out) {
  const int lane = threadIdx.x & 31;
  for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; r < n_rays;
       r += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const int64_t b = packed[2 * r];
    const int c = packed[2 * r + 1];
    for (int j = lane; j < c; j += 32) {
      ri_out[b + j] = ri_in[r * stride + j];
      ts_out[b + j] = ts_in[r * stride + j];
      te_out[b + j] = te_in[r * stride + j];
    }
  }
}

__global__ void grid_query_kernel(int64_t n, const float* __restrict__ x, GridView g,
                                  uint8_t* __restrict__ out) {
  load_roi(g);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    float p[3] = {x[3 * i], x[3 * i + 1], x[3 * i + 2]};
    out[i] = occupied_at(g, p) ? 1 : 0;
  }
}

// ---------------------------------------------------------------------------
// occupancy grid maintenance
// ---------------------------------------------------------------------------
// contract_inv for the three contraction types
// (NA/nerfacc/cuda/csrc/include/helpers_contraction.h:23-129).
__device__ __forceinline__ void contract_inv(const float lo[3], const float hi[3], int ctype,
                                             float u[3]) {
  if (ctype == SN_CONTRACTION_UN_BOUNDED_TANH) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      float v = atanhf(__fmaf_rn(u[d], 2.0f, -1.0f));
      v = fminf(fmaxf(v, -1e10f), 1e10f);
      u[d] = __fadd_rn(v, 0.5f);
    }
  } else if (ctype == SN_CONTRACTION_UN_BOUNDED_SPHERE) {
#pragma unroll
    for (int d = 0; d < 3; ++d) u[d] = __fmul_rn(__fsub_rn(u[d], 0.5f), 4.0f);
    float nsq = __fmaf_rn(u[2], u[2], __fmaf_rn(u[1], u[1], __fmul_rn(u[0], u[0])));
    float nrm = sqrtf(nsq);
    if (nrm > 1.0f) {
      float den = fmaxf(__fsub_rn(__fmul_rn(2.0f, nrm), __fmul_rn(1.0f, nsq)), 1e-10f);
#pragma unroll
      for (int d = 0; d < 3; ++d) u[d] = __fdiv_rn(u[d], den);
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) u[d] = __fmaf_rn(u[d], 0.5f, 0.5f);
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) u[d] = __fmaf_rn(u[d], __fsub_rn(hi[d], lo[d]), lo[d]);
}

__global__ void occ_points_kernel(int64_t n, const int64_t* __restrict__ cells,
                                  const float* __restrict__ jitter, int rx, int ry, int rz,
                                  const float* __restrict__ roi, int ctype, float* __restrict__ x) {
  float lo[3], hi[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    lo[d] = roi[d];
    hi[d] = roi[3 + d];
  }
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = cells ? cells[i] : i;
    const int64_t cz = c % rz, cy = (c / rz) % ry, cx = c / ((int64_t)ry * rz);
    float u[3];
    u[0] = __fdiv_rn(__fadd_rn((float)cx, jitter[3 * i + 0]), (float)rx);
    u[1] = __fdiv_rn(__fadd_rn((float)cy, jitter[3 * i + 1]), (float)ry);
    u[2] = __fdiv_rn(__fadd_rn((float)cz, jitter[3 * i + 2]), (float)rz);
    contract_inv(lo, hi, ctype, u);
    x[3 * i + 0] = u[0];
    x[3 * i + 1] = u[1];
    x[3 * i + 2] = u[2];
  }
}

constexpr int kReduceThreads = 512;

__global__ void __launch_bounds__(kReduceThreads)
occ_partial_sum(int64_t n, const float* __restrict__ occs, double* __restrict__ partial) {
  double s = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    s += (double)occs[i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ double ws[kReduceThreads / 32];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    double t = threadIdx.x < kReduceThreads / 32 ? ws[threadIdx.x] : 0.0;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (threadIdx.x == 0) partial[blockIdx.x] = t;
  }
}

__global__ void __launch_bounds__(kReduceThreads)
occ_threshold_kernel(int64_t n, const float* __restrict__ occs, const double* __restrict__ partial,
                     int n_partial, float thre, uint8_t* __restrict__ binary, float* mean_out) {
  __shared__ float s_thr;
  if (threadIdx.x < 32) {
    double t = 0.0;
    for (int k = threadIdx.x; k < n_partial; k += 32) t += partial[k];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (threadIdx.x == 0) {
      const float mean = (float)(t / (double)n);
      s_thr = fminf(mean, thre);
      if (mean_out && blockIdx.x == 0) *mean_out = mean;
    }
  }
  __syncthreads();
  const float thr = s_thr;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    binary[i] = occs[i] > thr ? 1 : 0;
}

// ---- device-side occupancy update (no host synchronisation) ----------------
// Query points of cells[i] (or cell i) with in-kernel jitter for i < *count.
__global__ void occ_points_n_kernel(int64_t cap, const int32_t* __restrict__ count,
                                    const int64_t* __restrict__ cells, uint64_t seed,
                                    const int32_t* __restrict__ stream_dev, int rx, int ry, int rz,
                                    const float* __restrict__ roi, int ctype, float* __restrict__ x) {
  const int64_t n = count ? min((int64_t)*count, cap) : cap;
  const uint64_t sid = stream_dev ? (uint64_t)(uint32_t)*stream_dev : 0ull;
  float lo[3], hi[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    lo[d] = roi[d];
    hi[d] = roi[3 + d];
  }
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = cells ? cells[i] : i;
    const int64_t cz = c % rz, cy = (c / rz) % ry, cx = c / ((int64_t)ry * rz);
    float u[3];
    u[0] = __fdiv_rn(__fadd_rn((float)cx, uniform01(seed, sid, 3 * (uint64_t)i + 0)), (float)rx);
    u[1] = __fdiv_rn(__fadd_rn((float)cy, uniform01(seed, sid, 3 * (uint64_t)i + 1)), (float)ry);
    u[2] = __fdiv_rn(__fadd_rn((float)cz, uniform01(seed, sid, 3 * (uint64_t)i + 2)), (float)rz);
    contract_inv(lo, hi, ctype, u);
    x[3 * i + 0] = u[0];
    x[3 * i + 1] = u[1];
    x[3 * i + 2] = u[2];
  }
}

// EMA update of the occupancy values (NA/nerfacc/grid.py:229-230:
// occs[indices] = max(occs[indices] * decay, occ)).  With cells == nullptr
// every cell appears once (the warm-up sweep) and one pass updates it in
// place.  Sampled cells may repeat, and every candidate must be formed from
// the cell's value before the update, so the sampled form takes three passes:
//   (1) vals[i] = max(occs[c] * decay, occ_i)       (reads occs only)
//   (2) occs[c] = vals[i]                            (a repeated cell keeps any one)
//   (3) atomicMax(occs[c], vals[i])                  (... then the largest)
// A repeated cell ends at max(old * decay, max_i occ_i): one of the values
// the reference's unordered index_put can store, and the one the scatter-max
// it names as intended gives.  occs >= 0 (an EMA of sigmoid values), so the
// float order equals the int order of the bit patterns.
__device__ __forceinline__ float occ_from_sdf(float sdf, float k) {
  // torch.sigmoid(-sdf * k) (models/renderer.py:56-60): 1 / (1 + exp(sdf * k))
  return 1.0f / (1.0f + expf(__fmul_rn(sdf, k)));
}

template <bool kFromSdf>
__global__ void occ_ema_value_kernel(int64_t cap, const int32_t* __restrict__ count,
                                     const int64_t* __restrict__ cells, const float* __restrict__ in,
                                     float k, float decay, float* __restrict__ occs,
                                     float* __restrict__ vals) {
  const int64_t n = count ? min((int64_t)*count, cap) : cap;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t c = cells ? cells[i] : i;
    const float occ = kFromSdf ? occ_from_sdf(in[i], k) : in[i];
    const float v = fmaxf(__fmul_rn(occs[c], decay), occ);
    if (cells)
      vals[i] = v;
    else
      occs[c] = v;
  }
}

__global__ void occ_ema_store_kernel(int64_t cap, const int32_t* __restrict__ count,
                                     const int64_t* __restrict__ cells, const float* __restrict__ vals,
                                     float* __restrict__ occs) {
  const int64_t n = count ? min((int64_t)*count, cap) : cap;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    occs[cells[i]] = vals[i];
}

__global__ void occ_ema_max_kernel(int64_t cap, const int32_t* __restrict__ count,
                                   const int64_t* __restrict__ cells, const float* __restrict__ vals,
                                   float* __restrict__ occs) {
  const int64_t n = count ? min((int64_t)*count, cap) : cap;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    atomicMax(reinterpret_cast<int*>(occs) + cells[i], __float_as_int(fmaxf(vals[i], 0.0f)));
}

// Launches the one-pass (all cells) or three-pass (sampled cells) update.
template <bool kFromSdf>
static int occ_ema_launch(int64_t cap, const int32_t* count, const int64_t* cells, const float* in,
                          float k, float decay, float* occs, float* vals, cudaStream_t st,
                          const char* what) {
  const unsigned g = stride_grid(cap, 256, 8);
  occ_ema_value_kernel<kFromSdf><<<g, 256, 0, st>>>(cap, count, cells, in, k, decay, occs, vals);
  if (!cells) return check_launch(what);
  occ_ema_store_kernel<<<g, 256, 0, st>>>(cap, count, cells, vals, occs);
  occ_ema_max_kernel<<<g, 256, 0, st>>>(cap, count, cells, vals, occs);
  return check_launch(what, 3);
}

__global__ void __launch_bounds__(kScanThreads)
u8_tile_count(const uint8_t* __restrict__ bits, int64_t n, int32_t* __restrict__ tile_sums) {
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i)
    if (base + i < n) s += bits[base + i] ? 1 : 0;
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ int ws[32];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    int t = ws[threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = t;
  }
}

__global__ void __launch_bounds__(kScanThreads)
u8_tile_compact(const uint8_t* __restrict__ bits, int64_t n, const int32_t* __restrict__ tile_off,
                int32_t* __restrict__ list) {
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int v[kScanItems], f[kScanItems];
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) f[i] = v[i] = (base + i < n && bits[base + i]) ? 1 : 0;
  block_exclusive_scan(v);
  const int off = tile_off[blockIdx.x];
#pragma unroll
  for (int i = 0; i < kScanItems; ++i)
    if (f[i]) list[off + v[i]] = (int32_t)(base + i);
}

// cells[0, n_uniform) uniform over the grid; then min(n_occ, n_uniform)
// occupied cells (all of them, or a uniform draw when there are more),
// as NA/nerfacc/grid.py:168-182 does; *count = total.
__global__ void occ_select_kernel(int64_t n_cells, int64_t n_uniform, const int32_t* __restrict__ list,
                                  const int32_t* __restrict__ n_occ_dev, uint64_t seed,
                                  const int32_t* __restrict__ stream_dev, int64_t* __restrict__ cells,
                                  int32_t* __restrict__ count) {
  const int64_t n_occ = *n_occ_dev;
  const uint64_t sid = stream_dev ? (uint64_t)(uint32_t)*stream_dev : 0ull;
  const int64_t n_take = n_occ < n_uniform ? n_occ : n_uniform;
  if (blockIdx.x == 0 && threadIdx.x == 0) *count = (int32_t)(n_uniform + n_take);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_uniform;
       i += (int64_t)gridDim.x * blockDim.x) {
    cells[i] = (int64_t)(uniform_u32(seed, sid ^ 0x5151u, (uint64_t)i) % (uint64_t)n_cells);
    if (i < n_take) {
      const int64_t j = n_occ > n_uniform
                            ? (int64_t)(uniform_u32(seed, sid ^ 0xA3A3u, (uint64_t)i) % (uint64_t)n_occ)
                            : i;
      cells[n_uniform + i] = list[j];
    }
  }
}

static int make_grid(GridView& g, const float* roi, const uint8_t* bits, int rx, int ry, int rz,
                     int ctype) {
  SN_REQUIRE(roi != nullptr, "roi is null");
  g.roi = roi;
  SN_REQUIRE(rx > 0 && ry > 0 && rz > 0, "grid resolution must be positive (%d,%d,%d)", rx, ry, rz);
  SN_REQUIRE(ctype >= 0 && ctype <= 2, "unknown contraction type %d", ctype);
  SN_REQUIRE(bits != nullptr, "grid_binary is null");
  g.res[0] = rx;
  g.res[1] = ry;
  g.res[2] = rz;
  g.bits = bits;
  g.ctype = ctype;
  return SN_OK;
}

}  // namespace sn

using namespace sn;

extern "C" {

const char* sn_version(void) { return "supernormal_gb300 0.1.0 (sm_103a)"; }

const char* sn_last_error(void) { return sn::g_err; }

uint64_t sn_kernel_launches(void) { return __atomic_load_n(&sn::g_launches, __ATOMIC_RELAXED); }

size_t sn_scan_workspace_bytes(int64_t n) {
  const int64_t n_tiles = (n + sn::kScanTile - 1) / sn::kScanTile;
  size_t b = (size_t)(n_tiles > 0 ? n_tiles : 1) * sizeof(int32_t);
  return (b + 255) & ~(size_t)255;
}

int sn_pack_counts(int64_t n, const int32_t* counts, int32_t* packed_info, int32_t* total,
                   void* workspace, void* stream) {
  SN_REQUIRE(n >= 0, "pack_counts: n < 0");
  SN_REQUIRE(n <= ((int64_t)1 << 31) - 1, "pack_counts: n too large");
  SN_REQUIRE(n == 0 || (counts && packed_info), "pack_counts: null buffer");
  return sn::pack_counts(n, counts, packed_info, total, workspace, as_stream(stream));
}

// sn_pack_counts without a caller workspace: the multi-tile scan's tile sums
// live in a file-scope device array, so the call allocates nothing.  Limit:
// kPackStaticMaxTiles tiles of kScanTile entries (16,777,216 entries, 16 KiB of
// scratch).  Nothing in the scratch has to start at zero (every tile sum is
// written by scan_tile_reduce before scan_tile_offsets reads it).  The scratch
// is one per device, so calls that overlap on the device (other streams or
// host threads) race on it.
int sn_pack_counts_n(int64_t cap, const int32_t* count, const int32_t* counts, int32_t* packed_info,
                     int32_t* total, void* workspace, void* stream) {
  SN_REQUIRE(cap >= 0, "pack_counts_n: cap < 0");
  SN_REQUIRE(cap <= ((int64_t)1 << 31) - 1, "pack_counts_n: cap too large");
  SN_REQUIRE(count != nullptr, "pack_counts_n: a device count is required");
  SN_REQUIRE(cap == 0 || (counts && packed_info), "pack_counts_n: null buffer");
  return sn::pack_counts(cap, counts, packed_info, total, workspace, as_stream(stream), count);
}

int sn_pack_counts_static(int64_t n, const int32_t* counts, int32_t* packed_info, int32_t* total,
                          void* stream) {
  SN_REQUIRE(n >= 0, "pack_counts_static: n < 0");
  SN_REQUIRE(n <= sn::kPackStaticMaxEntries,
             "pack_counts_static: n = %lld exceeds the static scratch limit of %lld entries",
             (long long)n, (long long)sn::kPackStaticMaxEntries);
  SN_REQUIRE(n == 0 || (counts && packed_info), "pack_counts_static: null buffer");
  int32_t* scratch = nullptr;
  SN_TRY(sn::pack_scratch_for_current_device(&scratch));
  return sn::pack_counts(n, counts, packed_info, total, scratch, as_stream(stream));
}

int sn_count_indices(int64_t n_samples, const int64_t* ray_indices, int64_t n_rays, int32_t* counts,
                     void* stream) {
  SN_REQUIRE(n_samples >= 0 && n_rays >= 0, "count_indices: negative size");
  cudaStream_t st = as_stream(stream);
  if (n_rays > 0 && cudaMemsetAsync(counts, 0, (size_t)n_rays * sizeof(int32_t), st) != cudaSuccess) {
    set_error("count_indices: memset failed");
    return SN_ERR_CUDA;
  }
  if (n_samples == 0) return SN_OK;
  count_indices_kernel<<<stride_grid(n_samples, 256, 8), 256, 0, st>>>(n_samples, ray_indices,
                                                                       n_rays, counts);
  return check_launch("count_indices");
}

size_t sn_pack_indices_workspace_bytes(int64_t n_rays) {
  const size_t counts = (size_t)(n_rays > 0 ? n_rays : 1) * sizeof(int32_t);
  return ((counts + 255) & ~(size_t)255) + sn_scan_workspace_bytes(n_rays);
}

int sn_pack_indices(int64_t n_samples, const int64_t* ray_indices, int64_t n_rays, int32_t* packed_info,
                    void* workspace, void* stream) {
  SN_REQUIRE(n_rays >= 0 && n_rays <= ((int64_t)1 << 31) - 1, "pack_indices: bad ray count");
  SN_REQUIRE(n_rays == 0 || (packed_info && workspace), "pack_indices: null buffer");
  int32_t* counts = reinterpret_cast<int32_t*>(workspace);
  SN_TRY(sn_count_indices(n_samples, ray_indices, n_rays, counts, stream));
  if (n_rays == 0) return SN_OK;
  const size_t scan = sn_pack_indices_workspace_bytes(n_rays) - sn_scan_workspace_bytes(n_rays);
  return sn_pack_counts(n_rays, counts, packed_info, nullptr, reinterpret_cast<char*>(workspace) + scan, stream);
}

int sn_unpack_info(int64_t n_rays, const int32_t* packed_info, int64_t n_samples,
                   int64_t* ray_indices, void* stream) {
  SN_REQUIRE(n_rays >= 0 && n_samples >= 0, "unpack_info: negative size");
  if (n_rays == 0 || n_samples == 0) return SN_OK;
  unpack_info_kernel<<<stride_grid(n_rays * 32, 256, 8), 256, 0, as_stream(stream)>>>(
      n_rays, packed_info, n_samples, ray_indices);
  return check_launch("unpack_info");
}

static int march_common(MarchArgs& a, int64_t n_rays, const float* rays_o, const float* rays_d,
                        const float* t_min, const float* t_max, const float* jitter,
                        const float* roi, const uint8_t* grid_binary, int rx, int ry, int rz,
                        int ctype, float step, float cone, int64_t max_iters, int32_t* status) {
  SN_REQUIRE(n_rays >= 0, "march: n_rays < 0");
  SN_REQUIRE(step > 0.0f && step < 1e30f, "march: step_size must be positive and finite (got %g)",
             (double)step);
  SN_REQUIRE(cone >= 0.0f && cone < 1e30f, "march: cone_angle must be >= 0 (got %g)", (double)cone);
  SN_REQUIRE(status != nullptr, "march: a device status word is required");
  SN_REQUIRE(roi != nullptr, "march: roi is null");
  memset(&a, 0, sizeof(a));
  SN_TRY(make_grid(a.grid, roi, grid_binary, rx, ry, rz, ctype));
  a.n_rays = n_rays;
  a.rays_o = rays_o;
  a.rays_d = rays_d;
  a.t_min = t_min;
  a.t_max = t_max;
  a.jitter = jitter;
  a.step = step;
  a.cone = cone;
  a.max_iters = max_iters > 0 ? max_iters : ((int64_t)1 << 24);
  a.status = status;
  return SN_OK;
}

// Count march; `blocks` (nullable) is filled first and shortens the walks.
static int launch_march_count(MarchArgs& a, uint32_t* blocks, int64_t max_samples, cudaStream_t st,
                              const char* what) {
  int launches = 1;
  if (blocks && a.grid.ctype == SN_CONTRACTION_AABB) {
    const BlockDims e = block_dims(a.grid);
    march_blocks_kernel<<<kBlockAxis * kBlockAxis / 8, 256, 0, st>>>(a.grid.bits, a.grid.res[0], a.grid.res[1],
                                                                     a.grid.res[2], e, blocks);
    a.blocks = blocks;
    ++launches;
  }
  const unsigned grid = div_up(a.n_rays * 32, 128);
  if (a.cone == 0.0f)
    launch_chained(march_warp_kernel<0, false>, grid, 128, 0, st, a, max_samples);
  else
    launch_chained(march_warp_kernel<0, true>, grid, 128, 0, st, a, max_samples);
  return check_launch(what, launches);
}

int sn_march_count(int64_t n_rays, const float* rays_o, const float* rays_d, const float* t_min,
                   const float* t_max, const float* jitter, const float* roi,
                   const uint8_t* grid_binary, int rx, int ry, int rz, int contraction_type,
                   float step_size, float cone_angle, int64_t max_iters, int32_t* num_steps,
                   int32_t* status, void* stream) {
  MarchArgs a;
  SN_TRY(march_common(a, n_rays, rays_o, rays_d, t_min, t_max, jitter, roi, grid_binary, rx, ry, rz,
                      contraction_type, step_size, cone_angle, max_iters, status));
  if (n_rays == 0) return SN_OK;
  a.num_steps = num_steps;
  return launch_march_count(a, nullptr, 0, as_stream(stream), "march_count");
}

size_t sn_march_runs_bytes(int64_t n_rays) {
  return (size_t)(n_rays > 0 ? n_rays : 1) * kMarchRuns * sizeof(float4) +
         (size_t)kBlockAxis * kBlockAxis * sizeof(uint32_t);
}

int sn_march_runs(int64_t n_rays, const float* rays_o, const float* rays_d, const float* t_min, const float* t_max,
                  const float* jitter, const float* roi, const uint8_t* grid_binary, int rx, int ry, int rz,
                  int contraction_type, float step_size, const float* step_size_dev, float cone_angle,
                  int64_t max_iters, int64_t max_samples, int32_t* num_steps, void* runs, int32_t* status,
                  void* stream) {
  MarchArgs a;
  SN_TRY(march_common(a, n_rays, rays_o, rays_d, t_min, t_max, jitter, roi, grid_binary, rx, ry, rz,
                      contraction_type, step_size, cone_angle, max_iters, status));
  if (n_rays == 0) return SN_OK;
  SN_REQUIRE(num_steps && runs, "march_runs: null output");
  SN_REQUIRE((reinterpret_cast<uintptr_t>(runs) & 15u) == 0, "march_runs: runs not 16-byte aligned");
  a.step_dev = step_size_dev;
  a.num_steps = num_steps;
  a.runs = reinterpret_cast<float4*>(runs);
  uint32_t* blocks = reinterpret_cast<uint32_t*>(a.runs + n_rays * kMarchRuns);
  return launch_march_count(a, n_rays >= kBlockRays ? blocks : nullptr, max_samples, as_stream(stream), "march_runs");
}

static int expand_args(MarchArgs& a, int64_t n_rays, const float* rays_o, const float* rays_d, const float* t_min,
                       const float* t_max, const float* jitter, const float* roi, const uint8_t* grid_binary, int rx,
                       int ry, int rz, int contraction_type, float step_size, const float* step_size_dev,
                       float cone_angle, int64_t max_iters, const void* runs, int64_t capacity, int64_t* ray_indices,
                       float* t_starts, float* t_ends, int32_t* status) {
  SN_TRY(march_common(a, n_rays, rays_o, rays_d, t_min, t_max, jitter, roi, grid_binary, rx, ry, rz,
                      contraction_type, step_size, cone_angle, max_iters, status));
  SN_REQUIRE(capacity >= 0, "march_expand: capacity < 0");
  if (n_rays == 0) return SN_OK;
  SN_REQUIRE(runs != nullptr, "march_expand: null input");
  SN_REQUIRE((reinterpret_cast<uintptr_t>(runs) & 15u) == 0, "march_expand: runs not 16-byte aligned");
  a.step_dev = step_size_dev;
  a.runs = const_cast<float4*>(reinterpret_cast<const float4*>(runs));
  a.capacity = capacity;
  a.ray_indices = ray_indices;
  a.t_starts = t_starts;
  a.t_ends = t_ends;
  return SN_OK;
}

static int launch_expand(const MarchArgs& a, bool counts, cudaStream_t st) {
  const auto fn = a.cone == 0.0f ? (counts ? march_expand_kernel<false, true> : march_expand_kernel<false, false>)
                                 : (counts ? march_expand_kernel<true, true> : march_expand_kernel<true, false>);
  launch_chained(fn, div_up(a.n_rays * 32, 128), 128, 0, st, a);
  return check_launch("march_expand");
}

int sn_march_expand(int64_t n_rays, const float* rays_o, const float* rays_d, const float* t_min, const float* t_max,
                    const float* jitter, const float* roi, const uint8_t* grid_binary, int rx, int ry, int rz,
                    int contraction_type, float step_size, const float* step_size_dev, float cone_angle,
                    int64_t max_iters, const int32_t* packed_info, const void* runs, int64_t capacity,
                    int64_t* ray_indices, float* t_starts, float* t_ends, int32_t* status, void* stream) {
  MarchArgs a;
  SN_TRY(expand_args(a, n_rays, rays_o, rays_d, t_min, t_max, jitter, roi, grid_binary, rx, ry, rz, contraction_type,
                     step_size, step_size_dev, cone_angle, max_iters, runs, capacity, ray_indices, t_starts, t_ends,
                     status));
  if (n_rays == 0) return SN_OK;
  SN_REQUIRE(packed_info != nullptr, "march_expand: null input");
  a.packed = packed_info;
  return launch_expand(a, false, as_stream(stream));
}

int sn_march_expand_counts(int64_t n_rays, const float* rays_o, const float* rays_d, const float* t_min,
                           const float* t_max, const float* jitter, const float* roi, const uint8_t* grid_binary,
                           int rx, int ry, int rz, int contraction_type, float step_size, const float* step_size_dev,
                           float cone_angle, int64_t max_iters, const int32_t* num_steps, int32_t* packed_info,
                           int32_t* total, void* scan_workspace, const void* runs, int64_t capacity,
                           int64_t* ray_indices, float* t_starts, float* t_ends, int32_t* status, void* stream) {
  MarchArgs a;
  SN_TRY(expand_args(a, n_rays, rays_o, rays_d, t_min, t_max, jitter, roi, grid_binary, rx, ry, rz, contraction_type,
                     step_size, step_size_dev, cone_angle, max_iters, runs, capacity, ray_indices, t_starts, t_ends,
                     status));
  if (n_rays == 0 || n_rays > kScanTile) {
    SN_TRY(sn_pack_counts(n_rays, num_steps, packed_info, total, scan_workspace, stream));
    a.packed = packed_info;
    return n_rays == 0 ? SN_OK : launch_expand(a, false, as_stream(stream));
  }
  SN_REQUIRE(num_steps && packed_info, "march_expand_counts: null buffer");
  SN_REQUIRE((reinterpret_cast<uintptr_t>(packed_info) & 7u) == 0, "march_expand_counts: packed_info not 8-byte aligned");
  a.num_steps = const_cast<int32_t*>(num_steps);
  a.packed_out = packed_info;
  a.total = total;
  return launch_expand(a, true, as_stream(stream));
}

int sn_march_padded(int64_t n_rays, const float* rays_o, const float* rays_d, const float* t_min,
                    const float* t_max, const float* jitter, const float* roi,
                    const uint8_t* grid_binary, int rx, int ry, int rz, int contraction_type,
                    float step_size, const float* step_size_dev, float cone_angle,
                    int64_t max_iters, int64_t slot_stride, int32_t* num_steps,
                    int64_t* ray_indices, float* t_starts, float* t_ends, int32_t* status,
                    void* stream) {
  MarchArgs a;
  SN_TRY(march_common(a, n_rays, rays_o, rays_d, t_min, t_max, jitter, roi, grid_binary, rx, ry, rz,
                      contraction_type, step_size, cone_angle, max_iters, status));
  SN_REQUIRE(slot_stride > 0, "march_padded: slot_stride must be positive");
  a.step_dev = step_size_dev;
  SN_REQUIRE(num_steps && ray_indices && t_starts && t_ends, "march_padded: null output");
  if (n_rays == 0) return SN_OK;
  a.num_steps = num_steps;
  a.capacity = n_rays * slot_stride;
  a.ray_indices = ray_indices;
  a.t_starts = t_starts;
  a.t_ends = t_ends;
  if (a.cone == 0.0f)
    march_warp_kernel<2, false><<<div_up(n_rays * 32, 128), 128, 0, as_stream(stream)>>>(a, slot_stride);
  else
    march_warp_kernel<2, true><<<div_up(n_rays * 32, 128), 128, 0, as_stream(stream)>>>(a, slot_stride);
  return check_launch("march_padded");
}

int sn_compact_padded(int64_t n_rays, int64_t slot_stride, const int32_t* packed_info,
                      const int64_t* ray_indices_in, const float* t_starts_in,
                      const float* t_ends_in, int64_t* ray_indices_out, float* t_starts_out,
                      float* t_ends_out, void* stream) {
  SN_REQUIRE(n_rays >= 0 && slot_stride > 0, "compact_padded: bad sizes");
  if (n_rays == 0) return SN_OK;
  compact_padded_kernel<<<stride_grid(n_rays * 32, 256, 8), 256, 0, as_stream(stream)>>>(
      n_rays, slot_stride, packed_info, ray_indices_in, t_starts_in, t_ends_in, ray_indices_out,
      t_starts_out, t_ends_out);
  return check_launch("compact_padded");
}

int sn_march_fill(int64_t n_rays, const float* rays_o, const float* rays_d, const float* t_min,
                  const float* t_max, const float* jitter, const float* roi,
                  const uint8_t* grid_binary, int rx, int ry, int rz, int contraction_type,
                  float step_size, float cone_angle, int64_t max_iters,
                  const int32_t* packed_info, int64_t capacity, int64_t* ray_indices,
                  float* t_starts, float* t_ends, int32_t* status, void* stream) {
  MarchArgs a;
  SN_TRY(march_common(a, n_rays, rays_o, rays_d, t_min, t_max, jitter, roi, grid_binary, rx, ry, rz,
                      contraction_type, step_size, cone_angle, max_iters, status));
  SN_REQUIRE(capacity >= 0, "march_fill: capacity < 0");
  if (n_rays == 0) return SN_OK;
  SN_REQUIRE(packed_info != nullptr, "march_fill: packed_info is null");
  a.packed = packed_info;
  a.capacity = capacity;
  a.ray_indices = ray_indices;
  a.t_starts = t_starts;
  a.t_ends = t_ends;
  if (a.cone == 0.0f)
    march_warp_kernel<1, false><<<div_up(n_rays * 32, 128), 128, 0, as_stream(stream)>>>(a, 0);
  else
    march_warp_kernel<1, true><<<div_up(n_rays * 32, 128), 128, 0, as_stream(stream)>>>(a, 0);
  return check_launch("march_fill");
}

int sn_grid_query(int64_t n, const float* samples, const float* roi, const uint8_t* grid_binary,
                  int rx, int ry, int rz, int contraction_type, uint8_t* out, void* stream) {
  SN_REQUIRE(n >= 0, "grid_query: n < 0");
  GridView g;
  memset(&g, 0, sizeof(g));
  SN_TRY(make_grid(g, roi, grid_binary, rx, ry, rz, contraction_type));
  if (n == 0) return SN_OK;
  grid_query_kernel<<<stride_grid(n, 256, 8), 256, 0, as_stream(stream)>>>(n, samples, g, out);
  return check_launch("grid_query");
}

int sn_occ_points(int64_t n, const int64_t* cells, const float* jitter, int rx, int ry, int rz,
                  const float* roi, int contraction_type, float* x_out, void* stream) {
  SN_REQUIRE(n >= 0, "occ_points: n < 0");
  SN_REQUIRE(rx > 0 && ry > 0 && rz > 0, "occ_points: bad resolution");
  SN_REQUIRE(contraction_type >= 0 && contraction_type <= 2, "occ_points: bad contraction");
  SN_REQUIRE(roi && jitter && x_out, "occ_points: null buffer");
  if (n == 0) return SN_OK;
  occ_points_kernel<<<stride_grid(n, 256, 8), 256, 0, as_stream(stream)>>>(
      n, cells, jitter, rx, ry, rz, roi, contraction_type, x_out);
  return check_launch("occ_points");
}

int sn_occ_ema_update(int64_t n, const int64_t* cells, const float* occ, float ema_decay,
                      float* occs, float* workspace, void* stream) {
  SN_REQUIRE(n >= 0, "occ_ema_update: n < 0");
  SN_REQUIRE(ema_decay >= 0.0f, "occ_ema_update: ema_decay < 0");
  SN_REQUIRE(occ && occs, "occ_ema_update: null buffer");
  SN_REQUIRE(!cells || workspace, "occ_ema_update: sampled cells need a workspace of n floats");
  if (n == 0) return SN_OK;
  return occ_ema_launch<false>(n, nullptr, cells, occ, 0.0f, ema_decay, occs, workspace,
                               as_stream(stream), "occ_ema_update");
}

size_t sn_occ_binarize_workspace_bytes(int64_t n_cells) {
  (void)n_cells;
  return (size_t)(4 * 1024) * sizeof(double);
}

int sn_occ_binarize(int64_t n_cells, const float* occs, float occ_thre, uint8_t* binary,
                    float* mean_out, void* workspace, void* stream) {
  SN_REQUIRE(n_cells > 0, "occ_binarize: n_cells must be > 0");
  SN_REQUIRE(workspace != nullptr, "occ_binarize: workspace required");
  cudaStream_t st = as_stream(stream);
  int nb = (int)stride_grid(n_cells, kReduceThreads, 4);
  if (nb > 4096) nb = 4096;
  double* partial = reinterpret_cast<double*>(workspace);
  occ_partial_sum<<<nb, kReduceThreads, 0, st>>>(n_cells, occs, partial);
  occ_threshold_kernel<<<stride_grid(n_cells, kReduceThreads, 4), kReduceThreads, 0, st>>>(
      n_cells, occs, partial, nb, occ_thre, binary, mean_out);
  return check_launch("occ_binarize", 2);
}

}  // extern "C"

extern "C" {

int sn_occ_points_n(int64_t cap, const int32_t* count, const int64_t* cells, uint64_t seed,
                    const int32_t* stream_counter, int rx, int ry, int rz, const float* roi,
                    int contraction_type, float* x_out, void* stream) {
  SN_REQUIRE(cap >= 0, "occ_points_n: cap < 0");
  SN_REQUIRE(rx > 0 && ry > 0 && rz > 0, "occ_points_n: bad resolution");
  SN_REQUIRE(contraction_type >= 0 && contraction_type <= 2, "occ_points_n: bad contraction");
  SN_REQUIRE(roi && x_out, "occ_points_n: null buffer");
  if (cap == 0) return SN_OK;
  occ_points_n_kernel<<<stride_grid(cap, 256, 8), 256, 0, as_stream(stream)>>>(
      cap, count, cells, seed, stream_counter, rx, ry, rz, roi, contraction_type, x_out);
  return check_launch("occ_points_n");
}

int sn_occ_ema_sdf(int64_t cap, const int32_t* count, const int64_t* cells, const float* sdf,
                   float sigmoid_k, float ema_decay, float* occs, float* workspace, void* stream) {
  SN_REQUIRE(cap >= 0, "occ_ema_sdf: cap < 0");
  SN_REQUIRE(sdf && occs, "occ_ema_sdf: null buffer");
  SN_REQUIRE(!cells || workspace, "occ_ema_sdf: sampled cells need a workspace of cap floats");
  if (cap == 0) return SN_OK;
  return occ_ema_launch<true>(cap, count, cells, sdf, sigmoid_k, ema_decay, occs, workspace,
                              as_stream(stream), "occ_ema_sdf");
}

size_t sn_occ_sample_workspace_bytes(int64_t n_cells) {
  const int64_t n_tiles = (n_cells + sn::kScanTile - 1) / sn::kScanTile;
  size_t b = (size_t)(n_tiles + 1) * sizeof(int32_t) + 256;   // tile offsets + total
  b += (size_t)n_cells * sizeof(int32_t);                      // occupied list
  return (b + 255) & ~(size_t)255;
}

int sn_occ_sample_cells(int64_t n_cells, const uint8_t* binary, int64_t n_uniform, uint64_t seed,
                        const int32_t* stream_counter, int64_t* cells, int32_t* count,
                        void* workspace, void* stream) {
  SN_REQUIRE(n_cells > 0 && n_uniform >= 0, "occ_sample_cells: bad sizes");
  SN_REQUIRE(binary && cells && count && workspace, "occ_sample_cells: null buffer");
  cudaStream_t st = as_stream(stream);
  const int64_t n_tiles = (n_cells + kScanTile - 1) / kScanTile;
  int32_t* tiles = reinterpret_cast<int32_t*>(workspace);
  int32_t* n_occ = tiles + n_tiles;
  int32_t* list = reinterpret_cast<int32_t*>(
      (reinterpret_cast<uintptr_t>(tiles + n_tiles + 1) + 255) & ~(uintptr_t)255);
  u8_tile_count<<<(unsigned)n_tiles, kScanThreads, 0, st>>>(binary, n_cells, tiles);
  scan_tile_offsets<<<1, kScanThreads, 0, st>>>(tiles, n_tiles, n_occ);
  u8_tile_compact<<<(unsigned)n_tiles, kScanThreads, 0, st>>>(binary, n_cells, tiles, list);
  occ_select_kernel<<<stride_grid(n_uniform > 0 ? n_uniform : 1, 256, 8), 256, 0, st>>>(
      n_cells, n_uniform, list, n_occ, seed, stream_counter, cells, count);
  return check_launch("occ_sample_cells", 4);
}

}  // extern "C"
