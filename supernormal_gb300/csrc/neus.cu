// Renderer glue of SuperNormal's patch-based NeuS training step
// (models/renderer.py:63-276) as device kernels:
//   * end-point bookkeeping: diff_mask = t_end != next t_start over the
//     flattened sample list (models/renderer.py:88-93, :151-154) and the
//     slot of every extra end evaluation;
//   * query-point builders for patch-centre samples (alpha_fn,
//     :80-98) and for all pixels of a patch via the marching plane
//     (t_pix = t_c * (d_c . n) / (d_pix . n), :146-159);
//   * NeuS SDF->alpha for the culling pass (:100-117);
//   * compaction of visible samples (NA/nerfacc/ray_marching.py:208-220);
//   * unit-sphere near/far with stratified jitter, mask binarisation.
// The fused per-patch render / loss / adjoint lives in patch.cu.
//
// Field query points are laid out as [S*P start points][E*P end points]:
// start (i, k) at i*P + k and the end of diff sample i at (S + slot_i)*P + k,
// which is the order the reference concatenates positions_all.
#include "neus_common.cuh"
#include "scan.cuh"
#include "weightnorm.cuh"

#include <string.h>

namespace sn {

// Whether sample i's end is evaluated by itself: t_ends[i] != t_starts[i+1]
// (the last sample compares with its own start).
__device__ __forceinline__ int end_differs(int64_t i, int64_t n, const float* ts, const float* te) {
  const float nxt = (i + 1 < n) ? ts[i + 1] : ts[i];
  return (__fsub_rn(te[i], nxt) != 0.0f) ? 1 : 0;
}

// diff[i] for i < min(*count, cap); entries past the count are not written.
__global__ void end_diff_kernel(int64_t cap, const int32_t* __restrict__ count,
                                const float* __restrict__ ts, const float* __restrict__ te,
                                int32_t* __restrict__ diff) {
  const int64_t n = count ? min((int64_t)*count, cap) : cap;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    diff[i] = end_differs(i, n, ts, te);
}

// The end slots in two launches, the second one the point builder that uses them
// (flags, a three-launch scan and the points were five, each 2-5 us at the sizes
// of an iteration: the launches, not their bytes, were the cost; 2,048 patches: 28 us
// for the centre and the patch points, now 18).  First: every
// sample's rank among the ends of its tile of kEndTile samples, and each tile's
// total.  The points' blocks then add the totals of the tiles before theirs, at
// most a few per thread, instead of a scan of them in a launch of its own.
constexpr int kEndTile = 1024;
__global__ void __launch_bounds__(kEndTile)
end_ranks_kernel(int64_t cap, const int32_t* __restrict__ count, const float* __restrict__ ts,
                 const float* __restrict__ te, int2* __restrict__ endp, int32_t* __restrict__ totals) {
  chained();
  __shared__ int ends[kEndTile / 32];
  const int64_t n = count ? min((int64_t)*count, cap) : cap;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t tile = blockIdx.x; tile * kEndTile < n; tile += gridDim.x) {
    const int64_t i = tile * kEndTile + threadIdx.x;
    const int diff = i < n ? end_differs(i, n, ts, te) : 0;
    const unsigned m = __ballot_sync(0xffffffffu, diff);
    if (lane == 0) ends[warp] = __popc(m);
    __syncthreads();
    const int before = __reduce_add_sync(0xffffffffu, lane < warp ? ends[lane] : 0);
    const int rank = before + __popc(m & ((1u << lane) - 1u));
    if (i < n) endp[i] = make_int2(rank, diff);
    if (threadIdx.x == kEndTile - 1) totals[tile] = rank + diff;
    __syncthreads();
  }
}

// Adding the totals before it is a few loads a thread for every block of an
// iteration's samples, but grows with their square: from this capacity on the totals
// are scanned in a launch of their own (the capacity decides, because the live count is
// on the device: an iteration's 2.1 M slots with 200,000 live samples stay below).
// Ranks and centre points, added / scanned: 1 M samples 13 / 16 us, 4 M 48 / 46, 16 M
// 222 / 180, 35 M 623 / 392 (flags, a scan of them and the points apart: 542).
constexpr int64_t kEndScanned = (int64_t)4096 * kEndTile;

// Ends of the tiles before `tile`, to every thread of a block of 256.  scanned:
// the totals are such sums already.
__device__ __forceinline__ int ends_before(const int32_t* __restrict__ totals, int64_t tile, bool scanned) {
  __shared__ int part[8];
  if (scanned) {
    __syncthreads();   // a barrier either way
    return totals[tile];
  }
  int s = 0;
  for (int64_t j = threadIdx.x; j < tile; j += 256) s += totals[j];
  s = __reduce_add_sync(0xffffffffu, s);
  __syncthreads();   // the last use of part
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  int sum = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) sum += part[w];
  return sum;
}

__device__ __forceinline__ void center_point(int64_t i, int64_t n, int2 ep, const int64_t* __restrict__ ridx,
                                             const float* __restrict__ ts, const float* __restrict__ te,
                                             const float* __restrict__ ro, const float* __restrict__ rd,
                                             float* __restrict__ xyz) {
  const int64_t r = ridx[i];
  const float t0 = ts[i], t1 = te[i];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float o = ro[3 * r + d], dd = rd[3 * r + d];
    xyz[3 * i + d] = __fadd_rn(o, __fmul_rn(dd, t0));
    if (ep.y) xyz[3 * (n + ep.x) + d] = __fadd_rn(o, __fmul_rn(dd, t1));
  }
}

// Centre-ray query points: starts then ends of diff samples.
__global__ void center_points_kernel(int64_t cap, const int32_t* __restrict__ count,
                                     const int64_t* __restrict__ ridx, const float* __restrict__ ts,
                                     const float* __restrict__ te, const float* __restrict__ ro,
                                     const float* __restrict__ rd, const int32_t* __restrict__ endp,
                                     const int32_t* __restrict__ n_ends, float* __restrict__ xyz,
                                     int32_t* __restrict__ q_out) {
  const int64_t n = count ? min((int64_t)*count, cap) : cap;
  if (blockIdx.x == 0 && threadIdx.x == 0 && q_out) q_out[0] = (int32_t)(n + *n_ends);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    center_point(i, n, reinterpret_cast<const int2*>(endp)[i], ridx, ts, te, ro, rd, xyz);
}

// The same from the ranks, which become the slots of end_packed; a block takes
// kCenterTile samples at a time.
constexpr int kCenterTile = 256;
__global__ void __launch_bounds__(256)
center_points_ranked_kernel(int64_t cap, const int32_t* __restrict__ count, const int64_t* __restrict__ ridx,
                            const float* __restrict__ ts, const float* __restrict__ te,
                            const float* __restrict__ ro, const float* __restrict__ rd,
                            const int32_t* __restrict__ totals, bool scanned, int2* __restrict__ endp,
                            int32_t* __restrict__ n_ends, float* __restrict__ xyz, int32_t* __restrict__ q_out) {
  chained();
  static_assert(kEndTile % kCenterTile == 0 && kCenterTile == 256, "one end tile, one sample a thread");
  const int64_t n = count ? min((int64_t)*count, cap) : cap;
  if (n == 0 && blockIdx.x == 0 && threadIdx.x == 0) {
    *n_ends = 0;
    if (q_out) *q_out = 0;
  }
  for (int64_t tile = blockIdx.x; tile * kCenterTile < n; tile += gridDim.x) {
    const int64_t i = tile * kCenterTile + threadIdx.x;
    int2 ep = make_int2(0, 0);
    if (i < n) ep = endp[i];
    const int before = ends_before(totals, tile / (kEndTile / kCenterTile), scanned);
    if (i < n) {
      ep.x += before;
      endp[i].x = ep.x;
      center_point(i, n, ep, ridx, ts, te, ro, rd, xyz);
      if (i == n - 1) {
        *n_ends = ep.x + ep.y;
        if (q_out) *q_out = (int32_t)(n + ep.x + ep.y);
      }
    }
  }
}

// Culling alpha at centre samples: sdf_next = end value if diff, else the next start.
__global__ void center_alpha_kernel(int64_t cap, const int32_t* __restrict__ count,
                                    const float* __restrict__ sdf, int sdf_stride,
                                    const int32_t* __restrict__ endp,
                                    const float* __restrict__ variance,
                                    float* __restrict__ alpha) {
  const int64_t n = count ? min((int64_t)*count, cap) : cap;
  const float inv_s = inv_s_from(variance);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int2 ep = reinterpret_cast<const int2*>(endp)[i];
    const float s0 = sdf[i * sdf_stride];
    const float s1 = ep.y ? sdf[(n + ep.x) * sdf_stride] : (i + 1 < n ? sdf[(i + 1) * sdf_stride] : s0);
    alpha[i] = neus_alpha(s0, s1, inv_s, nullptr, nullptr, nullptr);
  }
}

// The culling alpha and, from it, the visibility and visible count of every ray's
// samples: one warp per ray, the transmittance a warp product scan of (1 - alpha)
// with a carry between 32-sample chunks, as sn_visibility_from_alpha takes it.  The
// time is the longest ray's chain of chunks (loads, alpha, five scan steps), so the
// loads run ahead (a round's end values, whose addresses its slots give, one round,
// the rest two), kVisChunks chunks are scanned side by side, and a ray ends where its
// transmittance, which never grows, falls below eps.  In two launches (alpha, then
// visibility) they took 3.3 + 9 us at 2,048 rays of up to 1,000 samples; now 9.7.
constexpr int kVisChunks = 2;
__global__ void __launch_bounds__(256) center_visibility_kernel(
    int64_t n_rays, const int32_t* __restrict__ packed, int64_t cap, const int32_t* __restrict__ count,
    const float* __restrict__ sdf, int sdf_stride, const int2* __restrict__ endp,
    const float* __restrict__ variance, float eps, float thre, uint8_t* __restrict__ vis,
    int32_t* __restrict__ counts) {
  chained();
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int kRound = 32 * kVisChunks;
  const int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (r >= n_rays) return;  // whole warp
  const int64_t n = count ? min((int64_t)*count, cap) : cap;
  const int64_t base = packed[2 * r];
  const int steps = packed[2 * r + 1];
  // samples past the capacity have no field value
  const int live = (int)max(min((int64_t)steps, n - base), (int64_t)0);
  const float inv_s = inv_s_from(variance);
  struct Ahead {
    int2 ep;
    float s0, next;
  };
  const auto load = [&](int j, Ahead q[kVisChunks]) {
#pragma unroll
    for (int u = 0; u < kVisChunks; ++u) {
      q[u] = Ahead{make_int2(0, 0), 0.0f, 0.0f};
      if (j + 32 * u < live) {
        const int64_t i = base + j + 32 * u;
        q[u].ep = endp[i];
        q[u].s0 = sdf[i * sdf_stride];
        q[u].next = i + 1 < n ? sdf[(i + 1) * sdf_stride] : q[u].s0;
      }
    }
  };
  const auto ends = [&](const Ahead q[kVisChunks], float s1[kVisChunks]) {
#pragma unroll
    for (int u = 0; u < kVisChunks; ++u) s1[u] = q[u].ep.y ? sdf[(n + q[u].ep.x) * sdf_stride] : q[u].next;
  };
  Ahead cur[kVisChunks], next[kVisChunks];
  float s1[kVisChunks];
  load(lane, cur);
  load(kRound + lane, next);
  ends(cur, s1);
  float carry = 1.0f;
  int c = 0, j0 = 0;
  for (; j0 < live && carry >= eps; j0 += kRound) {
    Ahead after[kVisChunks];
    float s1_next[kVisChunks];
    load(j0 + 2 * kRound + lane, after);
    ends(next, s1_next);
    float al[kVisChunks], incl[kVisChunks];
#pragma unroll
    for (int u = 0; u < kVisChunks; ++u) {
      al[u] = neus_alpha(cur[u].s0, s1[u], inv_s, nullptr, nullptr, nullptr);
      incl[u] = j0 + 32 * u + lane < live ? __fsub_rn(1.0f, al[u]) : 1.0f;
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
      for (int u = 0; u < kVisChunks; ++u) {
        const float y = __shfl_up_sync(kAll, incl[u], o);
        if (lane >= o) incl[u] = __fmul_rn(y, incl[u]);
      }
#pragma unroll
    for (int u = 0; u < kVisChunks; ++u) {
      const int j = j0 + 32 * u + lane;
      float excl = __shfl_up_sync(kAll, incl[u], 1);
      if (lane == 0) excl = 1.0f;
      const float T = __fmul_rn(carry, excl);
      carry = __fmul_rn(carry, __shfl_sync(kAll, incl[u], 31));
      bool v = j < live && T >= eps;
      if (thre > 0.0f) v = v && (al[u] >= thre);
      if (j < live) vis[base + j] = v ? 1 : 0;
      c += __popc(__ballot_sync(kAll, v));
      cur[u] = next[u];
      next[u] = after[u];
      s1[u] = s1_next[u];
    }
  }
  for (int j = j0 + lane; j < live; j += 32) vis[base + j] = 0;
  if (lane == 0) counts[r] = c;
}

// Keep visible samples, preserving order: one warp per ray, a ballot per
// 32-sample chunk gives each visible sample its output slot.  kCompactChunks chunks
// are loaded together: a chunk at a time a ray of 1,000 samples waited 32 times for
// memory (8.8 us at 2,048 rays; now 4.8).
constexpr int kCompactChunks = 4;
// COUNTS: the output offsets are formed here, from the rays' visible counts.
// Samples at or past `count` and `cap` (a packed table may go past the capacity) are
// not read, and a ray writes no more than its output's slot holds.
struct CompactArgs {
  int64_t n_rays, cap;
  const int32_t* count;     // nullable
  const int32_t* pin;
  const uint8_t* vis;
  const int32_t* pout;      // the output's packed_info
  const int32_t* counts;    // COUNTS: instead of it, and where it and the total go
  int32_t *packed, *total;
  const int64_t* ridx;
  const float *ts, *te;
  int64_t* ridx_o;
  float *ts_o, *te_o;
};
template <bool COUNTS>
__global__ void __launch_bounds__(256) compact_kernel(CompactArgs a) {
  chained();
  const int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  int2 out;
  if constexpr (COUNTS) {
    out = packed_from_counts(a.counts, a.n_rays, a.packed, a.total);
    if (r >= a.n_rays) return;  // whole warp
  } else {
    if (r >= a.n_rays) return;  // whole warp
    out = make_int2(a.pout[2 * r], a.pout[2 * r + 1]);
  }
  const uint8_t* __restrict__ vis = a.vis;
  const int64_t* __restrict__ ridx = a.ridx;
  const float* __restrict__ ts = a.ts;
  const float* __restrict__ te = a.te;
  int64_t* __restrict__ ridx_o = a.ridx_o;
  float* __restrict__ ts_o = a.ts_o;
  float* __restrict__ te_o = a.te_o;
  const int64_t bi = a.pin[2 * r], bo = out.x;
  const int64_t n = a.count ? min((int64_t)*a.count, a.cap) : a.cap;
  const int steps = (int)min((int64_t)a.pin[2 * r + 1], n - bi), kept = out.y;
  int c = 0;
  for (int j0 = 0; j0 < steps && c < kept; j0 += 32 * kCompactChunks) {
    bool v[kCompactChunks];
    int at[kCompactChunks];
    int64_t ri[kCompactChunks];
    float t0[kCompactChunks], t1[kCompactChunks];
#pragma unroll
    for (int u = 0; u < kCompactChunks; ++u) {
      const int j = j0 + 32 * u + lane;
      v[u] = j < steps && vis[bi + j];
    }
#pragma unroll
    for (int u = 0; u < kCompactChunks; ++u) {
      const unsigned m = __ballot_sync(0xffffffffu, v[u]);
      at[u] = c + __popc(m & ((1u << lane) - 1u));
      v[u] = v[u] && at[u] < kept;
      c += __popc(m);
    }
#pragma unroll
    for (int u = 0; u < kCompactChunks; ++u) {
      const int j = j0 + 32 * u + lane;
      if (v[u]) {
        ri[u] = ridx[bi + j];
        t0[u] = ts[bi + j];
        t1[u] = te[bi + j];
      }
    }
#pragma unroll
    for (int u = 0; u < kCompactChunks; ++u) {
      if (v[u]) {
        ridx_o[bo + at[u]] = ri[u];
        ts_o[bo + at[u]] = t0[u];
        te_o[bo + at[u]] = t1[u];
      }
    }
  }
}

// Patch pixel expansion through the marching plane and query points: pixel k of
// sample i of n.
struct PatchPoints {
  int P, kc;
  const int64_t* pidx;
  const float *ts, *te, *ro, *rd, *pn;
  float *xyz, *tps, *tpe;
};
__device__ __forceinline__ void patch_point(const PatchPoints& a, int64_t i, int k, int64_t n, int2 ep) {
  const int64_t b = a.pidx[i], t = i * a.P + k;
  const float* nrm = a.pn + 3 * b;
  const float* dc = a.rd + (b * a.P + a.kc) * 3;
  const float* dp = a.rd + (b * a.P + k) * 3;
  const float* op = a.ro + (b * a.P + k) * 3;
  float dotc = __fmul_rn(dc[0], nrm[0]);
  dotc = __fadd_rn(dotc, __fmul_rn(dc[1], nrm[1]));
  dotc = __fadd_rn(dotc, __fmul_rn(dc[2], nrm[2]));
  float dotp = __fmul_rn(dp[0], nrm[0]);
  dotp = __fadd_rn(dotp, __fmul_rn(dp[1], nrm[1]));
  dotp = __fadd_rn(dotp, __fmul_rn(dp[2], nrm[2]));
  const float t0 = __fdiv_rn(__fmul_rn(a.ts[i], dotc), dotp);
  const float t1 = __fdiv_rn(__fmul_rn(a.te[i], dotc), dotp);
  float x0[3], x1[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    x0[d] = __fadd_rn(op[d], __fmul_rn(dp[d], t0));
    x1[d] = __fadd_rn(op[d], __fmul_rn(dp[d], t1));
  }
  // (stores only after the loads: they may alias)
  a.tps[t] = t0;
  a.tpe[t] = t1;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    a.xyz[3 * t + d] = x0[d];
    if (ep.y) a.xyz[3 * ((n + ep.x) * a.P + k) + d] = x1[d];
  }
}

__global__ void patch_points_kernel(int64_t cap, const int32_t* __restrict__ count, PatchPoints a,
                                    const int32_t* __restrict__ endp, const int32_t* __restrict__ n_ends,
                                    int32_t* __restrict__ q_out) {
  const int64_t n = count ? min((int64_t)*count, cap) : cap;
  if (blockIdx.x == 0 && threadIdx.x == 0 && q_out) q_out[0] = (int32_t)((n + *n_ends) * a.P);
  const int64_t total = n * a.P;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t / a.P;
    patch_point(a, i, (int)(t - i * a.P), n, reinterpret_cast<const int2*>(endp)[i]);
  }
}

// The same from the ranks of end_ranks_kernel, which become the slots of
// end_packed; a block takes kPatchTile samples at a time (a sample's pixels share
// its slot, so the slots go through shared memory).
constexpr int kPatchTile = 64;
__global__ void __launch_bounds__(256)
patch_points_ranked_kernel(int64_t cap, const int32_t* __restrict__ count, PatchPoints a,
                           const int32_t* __restrict__ totals, bool scanned, int2* __restrict__ endp,
                           int32_t* __restrict__ n_ends, int32_t* __restrict__ q_out) {
  chained();
  static_assert(kEndTile % kPatchTile == 0, "a patch tile lies in one end tile");
  __shared__ int2 slot[kPatchTile];
  const int64_t n = count ? min((int64_t)*count, cap) : cap;
  if (n == 0 && blockIdx.x == 0 && threadIdx.x == 0) {
    *n_ends = 0;
    if (q_out) *q_out = 0;
  }
  for (int64_t tile = blockIdx.x; tile * kPatchTile < n; tile += gridDim.x) {
    const int64_t i0 = tile * kPatchTile;
    const int len = (int)min((int64_t)kPatchTile, n - i0);
    int2 ep = make_int2(0, 0);
    if ((int)threadIdx.x < len) ep = endp[i0 + threadIdx.x];
    // (its barriers also end the previous tile's use of the slots)
    const int before = ends_before(totals, tile / (kEndTile / kPatchTile), scanned);
    if ((int)threadIdx.x < len) {
      ep.x += before;
      endp[i0 + threadIdx.x].x = ep.x;
      slot[threadIdx.x] = ep;
      if (i0 + threadIdx.x == n - 1) {
        *n_ends = ep.x + ep.y;
        if (q_out) *q_out = (int32_t)((n + ep.x + ep.y) * a.P);
      }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < len * a.P; t += 256) {
      const int j = t / a.P;
      patch_point(a, i0 + j, t - j * a.P, n, slot[j]);
    }
  }
}

// near/far of the unit-sphere chord for rays read with a stride
// (models/dataset_loader.py:279-297; NaN when the ray misses the sphere, so
// the marcher emits no samples for it), plus optional stratified jitter
// u in [0, 1) from the counter-based generator.
struct NearFar {
  int64_t n, stride;
  const float *ro, *rd;
  float *near, *far, *jitter;
  uint64_t seed;
  const int32_t* stream_dev;
  float *o_out, *d_out;
};
__device__ __forceinline__ void near_far_rays(const NearFar& a, int64_t first, int64_t step) {
  const uint64_t sid = a.stream_dev ? (uint64_t)(uint32_t)*a.stream_dev : 0ull;
  for (int64_t i = first; i < a.n; i += step) {
    const float* o = a.ro + i * a.stride;
    const float* d = a.rd + i * a.stride;
    if (a.o_out) {
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        a.o_out[3 * i + k] = o[k];
        a.d_out[3 * i + k] = d[k];
      }
    }
    const float dd = __fadd_rn(__fadd_rn(__fmul_rn(d[0], d[0]), __fmul_rn(d[1], d[1])), __fmul_rn(d[2], d[2]));
    const float od = __fadd_rn(__fadd_rn(__fmul_rn(o[0], d[0]), __fmul_rn(o[1], d[1])), __fmul_rn(o[2], d[2]));
    const float b = __fmul_rn(2.0f, od);
    const float oo = __fadd_rn(__fadd_rn(__fmul_rn(o[0], o[0]), __fmul_rn(o[1], o[1])), __fmul_rn(o[2], o[2]));
    const float c = __fsub_rn(oo, 1.0f);
    const float mid = __fdiv_rn(__fmul_rn(0.5f, -b), dd);
    const float h = __fdiv_rn(sqrtf(__fsub_rn(__fmul_rn(b, b), __fmul_rn(__fmul_rn(4.0f, dd), c))),
                              __fmul_rn(2.0f, dd));
    a.near[i] = __fsub_rn(mid, h);
    a.far[i] = __fadd_rn(mid, h);
    if (a.jitter) a.jitter[i] = uniform01(a.seed, sid, (uint64_t)i);
  }
}
__global__ void near_far_kernel(NearFar a) {
  near_far_rays(a, blockIdx.x * (int64_t)blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x);
}

__global__ void scale_count_kernel(const int32_t* __restrict__ in, int32_t mul, int32_t add,
                                   int32_t* __restrict__ out) {
  *out = *in * mul + add;
}

// mask := (mask > 0.5) as float, out = sum(mask) + 1e-5 (exp_runner.py:169-175).
// One block (no second pass); the sum of 0/1 values is exact in float below
// 2^24 elements, so the block size does not change it.
constexpr int kMaskThreads = 1024;
__device__ __forceinline__ void mask_prep_block(int64_t n, const float* __restrict__ mask_in,
                                                float* __restrict__ mask_out, float* __restrict__ mask_sum) {
  __shared__ float red[kMaskThreads / 32];
  float s = 0.0f;
  const int64_t n4 = (((uintptr_t)mask_in | (uintptr_t)mask_out) & 15) == 0 ? n / 4 : 0;
#pragma unroll 4
  for (int64_t i = threadIdx.x; i < n4; i += kMaskThreads) {
    float4 m = reinterpret_cast<const float4*>(mask_in)[i];
    m = make_float4(m.x > 0.5f ? 1.0f : 0.0f, m.y > 0.5f ? 1.0f : 0.0f, m.z > 0.5f ? 1.0f : 0.0f,
                    m.w > 0.5f ? 1.0f : 0.0f);
    reinterpret_cast<float4*>(mask_out)[i] = m;
    s += (m.x + m.y) + (m.z + m.w);
  }
  for (int64_t i = 4 * n4 + threadIdx.x; i < n; i += kMaskThreads) {
    const float m = mask_in[i] > 0.5f ? 1.0f : 0.0f;
    mask_out[i] = m;
    s += m;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.0f;
    for (int w = 0; w < kMaskThreads / 32; ++w) t += red[w];
    *mask_sum = t + 1e-5f;
  }
}
__global__ void __launch_bounds__(kMaskThreads)
mask_prep_kernel(int64_t n, const float* __restrict__ mask_in, float* __restrict__ mask_out,
                 float* __restrict__ mask_sum) {
  mask_prep_block(n, mask_in, mask_out, mask_sum);
}

// What an iteration starts with, none of it waiting for the rest: the masks (block
// 0), the effective weights of both layers with their gradients' zeros (a warp a
// row), and the centre rays' chords.  As six launches (two layers, two fills, masks,
// chords) they took 13-15 us of every iteration, 1-4 us each whatever their size;
// now 3.6 us with 256 patches and 5.7 us with 2,048.
struct StepBegin {
  int64_t n_mask;
  const float* mask_in;
  float *mask_out, *mask_sum;
  NearFar rays;
  sn_weightnorm_layer layer[2];
  int wn_blocks;
};
__global__ void __launch_bounds__(kMaskThreads) step_begin_kernel(const __grid_constant__ StepBegin a) {
  chained();
  const int b = (int)blockIdx.x - 1;
  if (b < 0) {
    mask_prep_block(a.n_mask, a.mask_in, a.mask_out, a.mask_sum);
  } else if (b < a.wn_blocks) {
    int r = b * (kMaskThreads / 32) + (threadIdx.x >> 5);
    for (int l = 0; l < 2; ++l) {
      if (r >= 0 && r < a.layer[l].rows) weightnorm_row(a.layer[l], r, threadIdx.x & 31, true);
      r -= a.layer[l].rows;
    }
  } else {
    near_far_rays(a.rays, (b - a.wn_blocks) * (int64_t)kMaskThreads + threadIdx.x,
                  (gridDim.x - 1 - a.wn_blocks) * (int64_t)kMaskThreads);
  }
}

// Copies of up to kCopyMax buffers in one launch (blockIdx.y is the buffer): 16
// bytes at a time where both sides allow it, else one float.
constexpr int kCopyMax = 8;
struct CopyArgs {
  float* dst[kCopyMax];
  const float* src[kCopyMax];
  int64_t n[kCopyMax];
};
__global__ void __launch_bounds__(256) copy_many_kernel(const __grid_constant__ CopyArgs a) {
  chained();
  float* dst = a.dst[blockIdx.y];
  const float* src = a.src[blockIdx.y];
  const int64_t n = a.n[blockIdx.y], t = blockIdx.x * (int64_t)256 + threadIdx.x, step = gridDim.x * (int64_t)256;
  const int64_t n4 = (((uintptr_t)dst | (uintptr_t)src) & 15) == 0 ? n / 4 : 0;
  for (int64_t i = t; i < n4; i += step) reinterpret_cast<float4*>(dst)[i] = reinterpret_cast<const float4*>(src)[i];
  for (int64_t i = 4 * n4 + t; i < n; i += step) dst[i] = src[i];
}

// One thread per patch pixel: world ray direction R normalize(K^-1 [x, y, 1]),
// V = rows (d, camera right, camera down) and V^-1 by the adjugate, in double
// and rounded once (models/dataset_loader.py:112-137), plus the ground-truth
// gathers and per-patch origin / plane normal (models/dataset_loader.py:223-277).
__global__ void gen_patches_kernel(int64_t n_patches, int ph, int pw, const int32_t* __restrict__ cx,
                                   const int32_t* __restrict__ cy, const int32_t* __restrict__ img, int H,
                                   int W, const double* __restrict__ kinv, const double* __restrict__ pose,
                                   const float* __restrict__ normals, const float* __restrict__ masks,
                                   float* __restrict__ rays_o, float* __restrict__ rays_d,
                                   float* __restrict__ plane_n, float* __restrict__ vinv,
                                   float* __restrict__ normal_out, float* __restrict__ mask_out) {
  const int P = ph * pw;
  const int64_t n = n_patches * P;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = i / P;
    const int r = (int)(i - b * P), yy = r / pw, xx = r - yy * pw;
    const int v = img[b];
    const int px = cx[b] + xx - pw / 2, py = cy[b] + yy - ph / 2;
    const double* K = kinv + 9 * v;
    const double* T = pose + 12 * v;   // rows of [R | t]
    double q[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) q[k] = K[3 * k] * px + K[3 * k + 1] * py + K[3 * k + 2];
    const double inv_norm = 1.0 / sqrt(q[0] * q[0] + q[1] * q[1] + q[2] * q[2]);
    double rw[3][3];   // rows d, right, down
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      rw[0][k] = (T[4 * k] * q[0] + T[4 * k + 1] * q[1] + T[4 * k + 2] * q[2]) * inv_norm;
      rw[1][k] = T[4 * k];
      rw[2][k] = T[4 * k + 1];
    }
    double c[3][3];    // c[j] = r(j+1) x r(j+2): column j of the adjugate
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const double* a = rw[(j + 1) % 3];
      const double* e = rw[(j + 2) % 3];
      c[j][0] = a[1] * e[2] - a[2] * e[1];
      c[j][1] = a[2] * e[0] - a[0] * e[2];
      c[j][2] = a[0] * e[1] - a[1] * e[0];
    }
    const double det = rw[0][0] * c[0][0] + rw[0][1] * c[0][1] + rw[0][2] * c[0][2];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      rays_d[3 * i + k] = (float)rw[0][k];
      rays_o[3 * i + k] = (float)T[4 * k + 3];
#pragma unroll
      for (int j = 0; j < 3; ++j) vinv[9 * i + 3 * k + j] = (float)(c[j][k] / det);
    }
    const int64_t pix = ((int64_t)v * H + py) * W + px;
    if (normals) {
#pragma unroll
      for (int k = 0; k < 3; ++k) normal_out[3 * i + k] = normals[3 * pix + k];
    }
    if (masks) mask_out[i] = masks[pix];
    if (r == 0) {
#pragma unroll
      for (int k = 0; k < 3; ++k) plane_n[3 * b + k] = (float)T[4 * k + 2];
    }
  }
}

static PatchPoints patch_points_args(int patch_h, int patch_w, const int64_t* pidx, const float* ts, const float* te,
                                     const float* ro, const float* rd, const float* pn, float* xyz, float* tps,
                                     float* tpe) {
  return PatchPoints{patch_h * patch_w, (patch_h / 2) * patch_w + patch_w / 2, pidx, ts, te, ro, rd, pn, xyz, tps, tpe};
}

}  // namespace sn

using namespace sn;

extern "C" {

int sn_end_diff(int64_t cap, const int32_t* count, const float* t_starts, const float* t_ends,
                int32_t* diff, void* stream) {
  SN_REQUIRE(cap >= 0, "end_diff: cap < 0");
  if (cap == 0) return SN_OK;
  end_diff_kernel<<<stride_grid(cap, 256, 8), 256, 0, as_stream(stream)>>>(cap, count, t_starts,
                                                                           t_ends, diff);
  return check_launch("end_diff");
}

int sn_center_points(int64_t cap, const int32_t* count, const int64_t* ray_indices,
                     const float* t_starts, const float* t_ends, const float* rays_o,
                     const float* rays_d, const int32_t* end_packed, const int32_t* n_ends,
                     float* xyz, int32_t* n_points, void* stream) {
  SN_REQUIRE(cap >= 0, "center_points: cap < 0");
  if (cap == 0) {  // no samples: no points
    if (n_points && cudaMemsetAsync(n_points, 0, sizeof(int32_t), as_stream(stream)) != cudaSuccess) {
      set_error("center_points: memset failed");
      return SN_ERR_CUDA;
    }
    return SN_OK;
  }
  SN_REQUIRE(n_ends != nullptr && end_packed != nullptr, "center_points: null end info");
  center_points_kernel<<<stride_grid(cap > 0 ? cap : 1, 256, 8), 256, 0, as_stream(stream)>>>(
      cap, count, ray_indices, t_starts, t_ends, rays_o, rays_d, end_packed, n_ends, xyz, n_points);
  return check_launch("center_points");
}

int sn_center_alpha(int64_t cap, const int32_t* count, const float* sdf, int sdf_stride,
                    const int32_t* end_packed, const float* variance, float* alpha, void* stream) {
  SN_REQUIRE(cap >= 0 && sdf_stride >= 1, "center_alpha: bad sizes");
  if (cap == 0) return SN_OK;
  center_alpha_kernel<<<stride_grid(cap, 256, 8), 256, 0, as_stream(stream)>>>(
      cap, count, sdf, sdf_stride, end_packed, variance, alpha);
  return check_launch("center_alpha");
}

int sn_compact_samples(int64_t n_rays, const int32_t* packed_in, const uint8_t* visibility,
                       const int32_t* packed_out, const int64_t* ray_indices,
                       const float* t_starts, const float* t_ends, int64_t* ray_indices_out,
                       float* t_starts_out, float* t_ends_out, void* stream) {
  SN_REQUIRE(n_rays >= 0, "compact: n_rays < 0");
  if (n_rays == 0) return SN_OK;
  launch_chained(compact_kernel<false>, div_up(n_rays * 32, 256), 256, 0, as_stream(stream),
      CompactArgs{n_rays, INT64_MAX, nullptr, packed_in, visibility, packed_out, nullptr, nullptr, nullptr,
                  ray_indices, t_starts, t_ends, ray_indices_out, t_starts_out, t_ends_out});
  return check_launch("compact_samples");
}

int sn_compact_counts(int64_t n_rays, const int32_t* packed_in, const uint8_t* visibility, const int32_t* counts,
                      int32_t* packed_out, int32_t* total, void* scan_workspace, const int64_t* ray_indices,
                      const float* t_starts, const float* t_ends, int64_t* ray_indices_out, float* t_starts_out,
                      float* t_ends_out, void* stream) {
  return sn_compact_counts_n(n_rays, packed_in, INT64_MAX, nullptr, visibility, counts, packed_out, total,
                             scan_workspace, ray_indices, t_starts, t_ends, ray_indices_out, t_starts_out, t_ends_out,
                             stream);
}

int sn_compact_counts_n(int64_t n_rays, const int32_t* packed_in, int64_t cap, const int32_t* count,
                        const uint8_t* visibility, const int32_t* counts, int32_t* packed_out, int32_t* total,
                        void* scan_workspace, const int64_t* ray_indices, const float* t_starts, const float* t_ends,
                        int64_t* ray_indices_out, float* t_starts_out, float* t_ends_out, void* stream) {
  SN_REQUIRE(n_rays >= 0 && cap >= 0, "compact: bad sizes");
  CompactArgs a{n_rays, cap, count, packed_in, visibility, packed_out, nullptr, nullptr, nullptr, ray_indices, t_starts,
                t_ends, ray_indices_out, t_starts_out, t_ends_out};
  if (n_rays == 0 || n_rays > kScanTile) {
    SN_TRY(sn_pack_counts(n_rays, counts, packed_out, total, scan_workspace, stream));
    if (n_rays == 0) return SN_OK;
    launch_chained(compact_kernel<false>, div_up(n_rays * 32, 256), 256, 0, as_stream(stream), a);
    return check_launch("compact_counts");
  }
  SN_REQUIRE(counts && packed_out, "compact_counts: null buffer");
  SN_REQUIRE(((uintptr_t)packed_out & 7) == 0, "compact_counts: packed_out not 8-byte aligned");
  a.counts = counts;
  a.packed = packed_out;
  a.total = total;
  launch_chained(compact_kernel<true>, div_up(n_rays * 32, 256), 256, 0, as_stream(stream), a);
  return check_launch("compact_counts");
}

int sn_patch_points(int64_t cap, const int32_t* count, int patch_h, int patch_w,
                    const int64_t* patch_indices, const float* t_starts, const float* t_ends,
                    const float* rays_o, const float* rays_d, const float* plane_normal,
                    const int32_t* end_packed, const int32_t* n_ends, float* xyz,
                    float* t_pix_starts, float* t_pix_ends, int32_t* n_points, void* stream) {
  SN_REQUIRE(cap >= 0 && patch_h >= 1 && patch_w >= 1, "patch_points: bad sizes");
  SN_REQUIRE(n_ends != nullptr && end_packed != nullptr, "patch_points: null end info");
  const PatchPoints a = patch_points_args(patch_h, patch_w, patch_indices, t_starts, t_ends, rays_o, rays_d,
                                          plane_normal, xyz, t_pix_starts, t_pix_ends);
  patch_points_kernel<<<stride_grid((cap > 0 ? cap : 1) * a.P, 256, 8), 256, 0, as_stream(stream)>>>(
      cap, count, a, end_packed, n_ends, n_points);
  return check_launch("patch_points");
}

size_t sn_end_ranks_workspace_bytes(int64_t cap) {
  const int64_t tiles = cap > 0 ? (cap + kEndTile - 1) / kEndTile : 1;
  return ((size_t)tiles * sizeof(int32_t) + 255) & ~(size_t)255;
}

int sn_end_ranks(int64_t cap, const int32_t* count, const float* t_starts, const float* t_ends,
                 int32_t* end_packed, void* workspace, void* stream) {
  SN_REQUIRE(cap >= 0 && cap <= ((int64_t)1 << 31) - 1, "end_ranks: bad capacity");
  if (cap == 0) return SN_OK;
  SN_REQUIRE(t_starts && t_ends && end_packed && workspace, "end_ranks: null buffer");
  SN_REQUIRE(((uintptr_t)end_packed & 7) == 0, "end_ranks: end_packed not 8-byte aligned");
  launch_chained(end_ranks_kernel, stride_grid(cap, kEndTile, 2), kEndTile, 0, as_stream(stream), cap, count,
      t_starts, t_ends, reinterpret_cast<int2*>(end_packed), reinterpret_cast<int32_t*>(workspace));
  SN_TRY(check_launch("end_ranks"));
  if (cap <= kEndScanned) return SN_OK;
  // (tiles past the live samples are not read: what is there is scanned for nothing)
  scan_tile_offsets<<<1, kScanThreads, 0, as_stream(stream)>>>(reinterpret_cast<int32_t*>(workspace),
                                                               (cap + kEndTile - 1) / kEndTile, nullptr);
  return check_launch("end_ranks");
}

int sn_center_points_ranked(int64_t cap, const int32_t* count, const int64_t* ray_indices,
                            const float* t_starts, const float* t_ends, const float* rays_o,
                            const float* rays_d, const void* workspace, int32_t* end_packed,
                            int32_t* n_ends, float* xyz, int32_t* n_points, void* stream) {
  SN_REQUIRE(cap >= 0 && cap <= ((int64_t)1 << 31) - 1, "center_points_ranked: bad capacity");
  SN_REQUIRE(n_ends != nullptr, "center_points_ranked: null n_ends");
  SN_REQUIRE(cap == 0 || (ray_indices && t_starts && t_ends && rays_o && rays_d && workspace && end_packed && xyz),
             "center_points_ranked: null buffer");
  SN_REQUIRE(((uintptr_t)end_packed & 7) == 0, "center_points_ranked: end_packed not 8-byte aligned");
  launch_chained(center_points_ranked_kernel, stride_grid(cap > 0 ? cap : 1, kCenterTile, 8), 256, 0,
      as_stream(stream), cap, count, ray_indices, t_starts, t_ends, rays_o, rays_d,
      reinterpret_cast<const int32_t*>(workspace), cap > kEndScanned, reinterpret_cast<int2*>(end_packed), n_ends,
      xyz, n_points);
  return check_launch("center_points_ranked");
}

int sn_patch_points_ranked(int64_t cap, const int32_t* count, int patch_h, int patch_w,
                           const int64_t* patch_indices, const float* t_starts, const float* t_ends,
                           const float* rays_o, const float* rays_d, const float* plane_normal,
                           const void* workspace, int32_t* end_packed, int32_t* n_ends, float* xyz,
                           float* t_pix_starts, float* t_pix_ends, int32_t* n_points, void* stream) {
  SN_REQUIRE(cap >= 0 && cap <= ((int64_t)1 << 31) - 1 && patch_h >= 1 && patch_w >= 1 &&
                 (int64_t)patch_h * patch_w <= 1 << 20,
             "patch_points_ranked: bad sizes");
  SN_REQUIRE(n_ends != nullptr, "patch_points_ranked: null n_ends");
  SN_REQUIRE(cap == 0 || (patch_indices && t_starts && t_ends && rays_o && rays_d && plane_normal && workspace &&
                          end_packed && xyz && t_pix_starts && t_pix_ends),
             "patch_points_ranked: null buffer");
  SN_REQUIRE(((uintptr_t)end_packed & 7) == 0, "patch_points_ranked: end_packed not 8-byte aligned");
  const PatchPoints a = patch_points_args(patch_h, patch_w, patch_indices, t_starts, t_ends, rays_o, rays_d,
                                          plane_normal, xyz, t_pix_starts, t_pix_ends);
  launch_chained(patch_points_ranked_kernel, stride_grid(cap > 0 ? cap : 1, kPatchTile, 8), 256, 0,
      as_stream(stream), cap, count, a, reinterpret_cast<const int32_t*>(workspace), cap > kEndScanned,
      reinterpret_cast<int2*>(end_packed), n_ends, n_points);
  return check_launch("patch_points_ranked");
}

int sn_center_visibility(int64_t n_rays, const int32_t* packed_info, int64_t cap, const int32_t* count,
                         const float* sdf, int sdf_stride, const int32_t* end_packed, const float* variance,
                         float early_stop_eps, float alpha_thre, uint8_t* visibility, int32_t* num_visible,
                         void* stream) {
  SN_REQUIRE(n_rays >= 0 && cap >= 0 && sdf_stride >= 1, "center_visibility: bad sizes");
  if (n_rays == 0) return SN_OK;
  SN_REQUIRE(packed_info && variance && num_visible, "center_visibility: null buffer");
  SN_REQUIRE(cap == 0 || (sdf && end_packed && visibility), "center_visibility: null buffer");
  SN_REQUIRE(((uintptr_t)end_packed & 7) == 0, "center_visibility: end_packed not 8-byte aligned");
  launch_chained(center_visibility_kernel, div_up(n_rays * 32, 256), 256, 0, as_stream(stream), n_rays, packed_info,
      cap, count, sdf, sdf_stride, reinterpret_cast<const int2*>(end_packed), variance, early_stop_eps, alpha_thre,
      visibility, num_visible);
  return check_launch("center_visibility");
}

int sn_step_begin(int64_t n_mask, const float* mask_in, float* mask_out, float* mask_sum, int64_t n_rays,
                  const float* rays_o, const float* rays_d, int64_t stride, float* near, float* far,
                  float* jitter, uint64_t seed, const int32_t* stream_counter, float* rays_o_out,
                  float* rays_d_out, const sn_weightnorm_layer* layer0, const sn_weightnorm_layer* layer1,
                  void* stream) {
  StepBegin a;
  memset(&a, 0, sizeof(a));
  SN_REQUIRE(n_mask >= 0 && n_rays >= 0 && stride >= 3, "step_begin: bad sizes");
  SN_REQUIRE(mask_sum && (n_mask == 0 || (mask_in && mask_out)), "step_begin: null mask");
  SN_REQUIRE(n_rays == 0 || (rays_o && rays_d && near && far), "step_begin: null buffer");
  SN_REQUIRE((rays_o_out == nullptr) == (rays_d_out == nullptr), "step_begin: give both ray copies or neither");
  SN_TRY(weightnorm_layers(layer0, layer1, false, a.layer));
  a.n_mask = n_mask;
  a.mask_in = mask_in;
  a.mask_out = mask_out;
  a.mask_sum = mask_sum;
  a.rays = NearFar{n_rays, stride, rays_o, rays_d, near, far, jitter, seed, stream_counter, rays_o_out, rays_d_out};
  a.wn_blocks = (int)div_up(a.layer[0].rows + a.layer[1].rows, kMaskThreads / 32);
  launch_chained(step_begin_kernel, 1 + a.wn_blocks + stride_grid(n_rays > 0 ? n_rays : 1, kMaskThreads, 1),
      kMaskThreads, 0, as_stream(stream), a);
  return check_launch("step_begin");
}

int sn_copy_many(int n_buffers, const sn_copy_buffer* buffers, void* stream) {
  SN_REQUIRE(n_buffers >= 0 && n_buffers <= kCopyMax, "copy_many: 0..%d buffers (got %d)", kCopyMax, n_buffers);
  SN_REQUIRE(n_buffers == 0 || buffers, "copy_many: null list");
  CopyArgs a;
  memset(&a, 0, sizeof(a));
  int64_t most = 0;
  for (int i = 0; i < n_buffers; ++i) {
    SN_REQUIRE(buffers[i].n >= 0, "copy_many: negative size");
    SN_REQUIRE(buffers[i].n == 0 || (buffers[i].dst && buffers[i].src), "copy_many: null buffer");
    SN_REQUIRE((((uintptr_t)buffers[i].dst | (uintptr_t)buffers[i].src) & 3) == 0, "copy_many: not 4-byte aligned");
    a.dst[i] = buffers[i].dst;
    a.src[i] = buffers[i].src;
    a.n[i] = buffers[i].n;
    most = buffers[i].n > most ? buffers[i].n : most;
  }
  if (most == 0) return SN_OK;
  launch_chained(copy_many_kernel, dim3((unsigned)stride_grid((most + 3) / 4, 256, 4), (unsigned)n_buffers), 256, 0,
      as_stream(stream), a);
  return check_launch("copy_many");
}

int sn_near_far_sphere(int64_t n, const float* rays_o, const float* rays_d, int64_t stride,
                       float* near, float* far, float* jitter, uint64_t seed,
                       const int32_t* stream_counter, float* rays_o_out, float* rays_d_out,
                       void* stream) {
  SN_REQUIRE(n >= 0 && stride >= 3, "near_far_sphere: bad sizes");
  SN_REQUIRE(rays_o && rays_d && near && far, "near_far_sphere: null buffer");
  SN_REQUIRE((rays_o_out == nullptr) == (rays_d_out == nullptr),
             "near_far_sphere: give both ray copies or neither");
  if (n == 0) return SN_OK;
  near_far_kernel<<<stride_grid(n, 256, 8), 256, 0, as_stream(stream)>>>(
      NearFar{n, stride, rays_o, rays_d, near, far, jitter, seed, stream_counter, rays_o_out, rays_d_out});
  return check_launch("near_far_sphere");
}

int sn_gen_patches(int64_t n_patches, int patch_h, int patch_w, const int32_t* cx, const int32_t* cy,
                   const int32_t* img, int n_views, int H, int W, const double* kinv, const double* pose,
                   const float* normals, const float* masks, float* rays_o, float* rays_d, float* plane_n,
                   float* vinv, float* normal_out, float* mask_out, void* stream) {
  SN_REQUIRE(n_patches >= 0 && patch_h >= 1 && patch_w >= 1 && n_views >= 1 && H >= patch_h && W >= patch_w,
             "gen_patches: bad sizes");
  SN_REQUIRE(cx && cy && img && kinv && pose && rays_o && rays_d && plane_n && vinv, "gen_patches: null buffer");
  SN_REQUIRE(!normals || normal_out, "gen_patches: normals given without normal_out");
  SN_REQUIRE(!masks || mask_out, "gen_patches: masks given without mask_out");
  if (n_patches == 0) return SN_OK;
  gen_patches_kernel<<<stride_grid(n_patches * patch_h * patch_w, 256, 8), 256, 0, as_stream(stream)>>>(
      n_patches, patch_h, patch_w, cx, cy, img, H, W, kinv, pose, normals, masks, rays_o, rays_d, plane_n, vinv,
      normal_out, mask_out);
  return check_launch("gen_patches");
}

int sn_scale_count(const int32_t* in, int32_t mul, int32_t add, int32_t* out, void* stream) {
  SN_REQUIRE(in && out, "scale_count: null buffer");
  scale_count_kernel<<<1, 1, 0, as_stream(stream)>>>(in, mul, add, out);
  return check_launch("scale_count");
}

int sn_mask_prep(int64_t n, const float* mask_in, float* mask_out, float* mask_sum, void* stream) {
  SN_REQUIRE(n >= 0, "mask_prep: n < 0");
  mask_prep_kernel<<<1, kMaskThreads, 0, as_stream(stream)>>>(n, mask_in, mask_out, mask_sum);
  return check_launch("mask_prep");
}

}  // extern "C"
