// SDF field: multi-resolution hash-grid encoding + one-hidden-layer MLP.
//
// Encoding: Instant-NGP multiresolution hash encoding (Mueller et al. 2022)
// with tiny-cuda-nn's conventions as used by SuperNormal's
// `tcnn.Encoding(3, {otype: HashGrid, ...})` (models/fields.py:26,78):
//   scale_l = 2^(l*log2(per_level_scale)) * base_resolution - 1
//   resolution_l = ceil(scale_l) + 1
//   pos = fma(scale_l, x, 0.5); cell = floor(pos); frac = pos - cell
//   dense index (cell_x + cell_y*res + cell_z*res^2) when res^3 fits the
//   level, else the XOR prime hash (1, 2654435761, 805459861); both taken
//   modulo the level size in uint32 arithmetic (so SuperNormal's [-1,1]
//   inputs wrap exactly as they do there), trilinear weights over the 8
//   corners in corner order 0..7.
// Table layout: entry-major, F features contiguous per entry, levels
// concatenated at offsets[l] (the tcnn `params` layout).
//
// MLP: SDFNetwork with n_layers = 1 and input_concat
// (models/fields.py:76-99): in = [x, enc], h = W0 in + b0,
// a = softplus_beta(h), y = W1 a + b1, with W0/W1 the weight-normed
// matrices.  Levels at or beyond `active_levels` are the encoding features
// SuperNormal masks to zero (bandwidth, models/fields.py:81-83); their
// gather and gradient are skipped, which is exact because the mask
// multiplies them by zero.
#include "cluster.cuh"
#include "field_common.cuh"
#include "weightnorm.cuh"

#include <math.h>
#include <string.h>

namespace sn {

// --- standalone encoding (tcnn.Encoding forward / backward) -----------------
__global__ void hashgrid_fwd_kernel(int64_t n, const float* __restrict__ x,
                                    const float* __restrict__ table, GridDev g, int active,
                                    float* __restrict__ out) {
  const int64_t total = n * g.L;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = t / g.L;
    const int l = (int)(t - p * g.L);
    float e0 = 0.0f, e1 = 0.0f;
    if (l < active) {
      const float xp[3] = {x[3 * p], x[3 * p + 1], x[3 * p + 2]};
      encode_level(table, g, l, xp, e0, e1);
    }
    reinterpret_cast<float2*>(out)[t] = make_float2(e0, e1);
  }
}

__global__ void hashgrid_bwd_kernel(int64_t n, const float* __restrict__ x,
                                    const float* __restrict__ gout, GridDev g, int active,
                                    float* __restrict__ gtable) {
  const int64_t total = n * g.L;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = t / g.L;
    const int l = (int)(t - p * g.L);
    if (l >= active) continue;
    const float xp[3] = {x[3 * p], x[3 * p + 1], x[3 * p + 2]};
    const float2 go = reinterpret_cast<const float2*>(gout)[t];
    LevelCorners c;
    level_corners(g, l, xp, c);
    float2* gt2 = reinterpret_cast<float2*>(gtable);
#pragma unroll
    for (int k = 0; k < 8; ++k) atomicAdd(gt2 + c.idx[k], make_float2(c.w[k] * go.x, c.w[k] * go.y));
  }
}

// --- weight normalisation (torch.nn.utils.weight_norm, dim=0) ----------------
// A warp a row; two layers in one launch (blockIdx.y), because a launch costs its
// 2-3 us whatever its 65 rows do.
struct WeightNormArgs {
  sn_weightnorm_layer layer[2];
};
template <bool ADJOINT>
__global__ void __launch_bounds__(128) weightnorm_kernel(const __grid_constant__ WeightNormArgs a) {
  chained();
  const sn_weightnorm_layer& l = a.layer[blockIdx.y];
  const int r = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (r >= l.rows) return;  // whole warp
  if (ADJOINT)
    weightnorm_row_bwd(l, r, threadIdx.x & 31);
  else
    weightnorm_row(l, r, threadIdx.x & 31, false);
}

// Up to eight buffers to be cleared in one launch.
constexpr int kClearMax = 8;
struct ClearArgs {
  float* dst[kClearMax];
  int64_t n[kClearMax];
  int count;
  void add(float* p, int64_t len) {
    if (p == nullptr || len <= 0) return;
    dst[count] = p;
    n[count++] = len;
  }
};

// Column sums of the output gradients, (n, cols) with at most kDoutMax columns: the
// output biases' gradient.  Half a million terms that cancel to a ten-thousandth of
// their size are the rule here, and summed in float by atomics, whose order changes
// from call to call, they left the bias 1e-7 to 1e-5 off.  So: one cluster, sums in
// float with their rounding errors beside them, added in a fixed order (in double, of
// which the chip does two a cycle and SM, the blocks' sums only: with a double sum a
// thread an iteration of 256 patches took 147 us, now 140).  A thread's terms are VEC
// neighbouring floats, `period` threads after which the columns repeat apart.
constexpr int kSumThreads = 1024, kSumCluster = 8, kSumAhead = 8;
// (s, e): s is the float sum, s + e the sum to about 48 bits (s alone where s is
// infinite or NaN).
__device__ __forceinline__ float2 pair_add(float2 a, float2 b) {
  const float s = __fadd_rn(a.x, b.x), c = __fsub_rn(s, a.x);   // Knuth's two-sum
  const float e = __fadd_rn(__fsub_rn(a.x, __fsub_rn(s, c)), __fsub_rn(b.x, c));
  return make_float2(s, __fadd_rn(e, __fadd_rn(a.y, b.y)));
}
struct ColumnSums {
  int64_t cap;
  const int32_t* count;
  const float* g;
  int cols, period;
  float* out;
  int rows;   // of out that are written (zeros behind the sums); 0: the sums are added
};
// A cluster of kSumCluster blocks; every thread takes part.
template <int VEC, bool ONE>
__device__ __forceinline__ void column_sums(const ColumnSums& a) {
  cluster_arrive();
  const float* __restrict__ g = a.g;
  const int cols = a.cols;
  __shared__ float2 sums[ONE ? kSumThreads / 32 : VEC * kSumThreads];
  __shared__ double parts[kSumCluster][kDoutMax];   // of the first block
  const int t = threadIdx.x, active = kSumThreads / a.period * a.period;
  const uint32_t rank = cluster_rank();
  const int64_t total = (a.count ? max(min((int64_t)*a.count, a.cap), (int64_t)0) : a.cap) * cols;
  const int64_t items = total / VEC, step = (int64_t)kSumCluster * active;
  float2 s[VEC];
#pragma unroll
  for (int i = 0; i < VEC; ++i) s[i] = make_float2(0.0f, 0.0f);
  for (int64_t v = t < active ? rank * (int64_t)active + t : items; v < items; v += kSumAhead * step) {
    float x[kSumAhead][VEC];
#pragma unroll
    for (int u = 0; u < kSumAhead; ++u) {
      const int64_t w = v + u * step;
      if constexpr (VEC == 4) {
        const float4 q = w < items ? reinterpret_cast<const float4*>(g)[w] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        x[u][0] = q.x, x[u][1] = q.y, x[u][2] = q.z, x[u][3] = q.w;
      } else {
        x[u][0] = w < items ? g[w] : 0.0f;
      }
    }
#pragma unroll
    for (int u = 0; u < kSumAhead; ++u)
#pragma unroll
      for (int i = 0; i < VEC; ++i) s[i] = pair_add(s[i], make_float2(x[u][i], 0.0f));
  }
  if constexpr (ONE) {
#pragma unroll
    for (int i = 1; i < VEC; ++i) s[0] = pair_add(s[0], s[i]);
    for (int half = 0; half < 2; ++half) {   // over the warp's lanes, then over the warps
      if (half == 0 || t < 32) {
        if (half) s[0] = sums[t];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
          s[0] = pair_add(s[0], make_float2(__shfl_xor_sync(0xffffffffu, s[0].x, o), __shfl_xor_sync(0xffffffffu, s[0].y, o)));
        if ((t & 31) == 0) sums[t >> 5] = s[0];
      }
      __syncthreads();
    }
  } else {
#pragma unroll
    for (int i = 0; i < VEC; ++i)
      if (t < active) sums[VEC * t + i] = s[i];
    __syncthreads();
    for (int rows = VEC * active / cols; rows > 1;) {   // pairs of rows of `cols` sums, until one is left
      const int half = (rows + 1) / 2;
      for (int e = t; e < (rows - half) * cols; e += kSumThreads) sums[e] = pair_add(sums[e], sums[e + half * cols]);
      __syncthreads();
      rows = half;
    }
  }
  cluster_wait();   // the first block runs
  if (t < cols) st_cluster(&parts[rank][t], 0, (double)sums[t].x + (isfinite(sums[t].x) ? (double)sums[t].y : 0.0));
  cluster_arrive();
  cluster_wait();
  if (rank == 0 && t < cols) {
    double d = 0.0;
    for (int b = 0; b < kSumCluster; ++b) d += parts[b][t];
    for (int64_t e = items * VEC; e < total; ++e)
      if (e % cols == t) d += (double)g[e];
    if (a.rows)
      a.out[t] = (float)d;
    else
      atomicAdd(a.out + t, (float)d);
  }
  if (rank == 0 && t >= cols && t < a.rows) a.out[t] = 0.0f;
}
template <int VEC, bool ONE>
__global__ void __cluster_dims__(kSumCluster, 1, 1) __launch_bounds__(kSumThreads)
column_sums_kernel(const __grid_constant__ ColumnSums a) {
  chained();
  column_sums<VEC, ONE>(a);
}
// With what a backward clears before it: the first cluster sums meanwhile (500,003
// points and a table of 12.6 M floats: 16.5 us, apart 9.5 and 12.7).
template <int VEC, bool ONE>
__global__ void __cluster_dims__(kSumCluster, 1, 1) __launch_bounds__(kSumThreads)
clear_and_sum_kernel(const __grid_constant__ ClearArgs c, const __grid_constant__ ColumnSums a) {
  chained();
  if (blockIdx.x < kSumCluster) {
    if (a.out) column_sums<VEC, ONE>(a);
    return;
  }
  const int64_t t = (blockIdx.x - kSumCluster) * (int64_t)kSumThreads + threadIdx.x;
  const int64_t step = (gridDim.x - kSumCluster) * (int64_t)kSumThreads;
  for (int b = 0; b < c.count; ++b) {
    float* dst = c.dst[b];
    const int64_t n = c.n[b], n4 = ((uintptr_t)dst & 15) == 0 ? n / 4 : 0;
    for (int64_t i = t; i < n4; i += step) reinterpret_cast<float4*>(dst)[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int64_t i = 4 * n4 + t; i < n; i += step) dst[i] = 0.0f;
  }
}
ColumnSums make_sums(int64_t cap, const int32_t* count, const float* g, int cols, float* out, int rows, bool& quads) {
  quads = (reinterpret_cast<uintptr_t>(g) & 15u) == 0;
  const int period = !quads ? cols : cols / ((cols & 3) == 0 ? 4 : (cols & 1) == 0 ? 2 : 1);   // quads: lcm(4, cols) / 4
  return ColumnSums{cap, count, g, cols, period, out, rows};
}
int add_bias_grad(const FieldArgs& a, const float* g, int cols, float* grad_b1, cudaStream_t st) {
  if (g == nullptr || grad_b1 == nullptr) return SN_OK;
  bool quads;
  const ColumnSums s = make_sums(a.cap, a.count, g, cols, grad_b1, 0, quads);
  const auto fn = quads ? (cols == 1 ? column_sums_kernel<4, true> : column_sums_kernel<4, false>)
                        : (cols == 1 ? column_sums_kernel<1, true> : column_sums_kernel<1, false>);
  launch_chained(fn, kSumCluster, kSumThreads, 0, st, s);
  return check_launch("bias_grad");
}

// The gradients that a field backward of n points adds to, cleared, and the output
// biases' written: the column sums of g (n, cols).
int begin_field_grads(const sn_weightnorm_layer& l0, const sn_weightnorm_layer& l1, float* grad_table, int64_t n_table,
                      float* grad_b0, float* grad_b1, int64_t n, const float* g, int cols, cudaStream_t st) {
  ClearArgs a;
  memset(&a, 0, sizeof(a));
  a.add(grad_table, n_table);
  a.add(l0.grad_w, (int64_t)l0.rows * l0.cols);
  if (l1.grad_w_sums)
    a.add(reinterpret_cast<float*>(l1.grad_w_sums), 2 * (int64_t)l1.rows * l1.cols);
  else
    a.add(l1.grad_w, (int64_t)l1.rows * l1.cols);
  a.add(grad_b0, l0.rows);
  const bool sum = grad_b1 && g && n > 0 && cols >= 1 && cols <= l1.rows && l1.rows <= kDoutMax;
  if (!sum) a.add(grad_b1, l1.rows);
  if (a.count == 0 && !sum) return SN_OK;
  int64_t most = 1;
  for (int i = 0; i < a.count; ++i) most = a.n[i] > most ? a.n[i] : most;
  bool quads;
  const ColumnSums s = make_sums(n, nullptr, g, sum ? cols : 1, sum ? grad_b1 : nullptr, l1.rows, quads);
  const auto fn = quads ? (s.cols == 1 ? clear_and_sum_kernel<4, true> : clear_and_sum_kernel<4, false>)
                        : (s.cols == 1 ? clear_and_sum_kernel<1, true> : clear_and_sum_kernel<1, false>);
  const unsigned blocks = (unsigned)stride_grid((most + 3) / 4, kSumThreads, 2);
  launch_chained(fn, kSumCluster + (blocks + kSumCluster - 1) / kSumCluster * kSumCluster, kSumThreads, 0, st, a, s);
  return check_launch("field_grads");
}

int check_wn(const sn_mlp_desc* mlp, const sn_weightnorm_layer* l0, const sn_weightnorm_layer* l1) {
  SN_REQUIRE(mlp && l0 && l1, "field_wn: null descriptor");
  SN_REQUIRE(l0->rows == mlp->d_hidden && l0->cols == mlp->d_in && l1->rows == mlp->d_out && l1->cols == mlp->d_hidden,
             "field_wn: the layers do not fit the network");
  SN_REQUIRE(l0->w == mlp->w0 && l1->w == mlp->w1, "field_wn: the layers' weights are not the network's");
  SN_REQUIRE(!l0->grad_w_sums && (!l1->grad_w_sums || l1->grad_w), "field_wn: sums in double are the output layer's");
  SN_REQUIRE((reinterpret_cast<uintptr_t>(l1->grad_w_sums) & 7u) == 0, "field_wn: grad_w_sums not 8-byte aligned");
  return SN_OK;
}

int make_grid_dev(const sn_grid_desc* d, GridDev& g) {
  SN_REQUIRE(d != nullptr, "grid descriptor is null");
  SN_REQUIRE(d->n_features == kF, "only %d features per level are supported (got %d)", kF,
             d->n_features);
  if (d->n_levels < 1 || d->n_levels > kMaxL) {
    set_error("1..%d levels supported (got %d)", kMaxL, d->n_levels);
    return SN_ERR_UNSUPPORTED;
  }
  memset(&g, 0, sizeof(g));
  g.L = d->n_levels;
  for (int l = 0; l < g.L; ++l) {
    const uint32_t size = d->offsets[l + 1] - d->offsets[l];
    SN_REQUIRE(size > 0, "empty level %d", l);
    LevelDev& v = g.lv[l];
    const uint64_t r = d->resolutions[l];
    const bool dense = r * r * r <= (uint64_t)size, pow2 = (size & (size - 1)) == 0;
    v.scale = d->scales[l];
    v.offset = d->offsets[l];
    v.size = size;
    v.kind = dense ? (r * r + r < size ? kDense : kGeneralDense) : (pow2 ? kHashed : kGeneralHash);
    v.my = dense ? d->resolutions[l] : 2654435761u;
    v.mz = dense ? d->resolutions[l] * d->resolutions[l] : 805459861u;
    int lg = 0;
    while (((uint64_t)1 << lg) < size) ++lg;
    const uint64_t m = (((uint64_t)1 << 32) * (((uint64_t)1 << lg) - size)) / size + 1;
    v.magic = (uint32_t)m;
    v.shifts = (uint32_t)(lg < 1 ? lg : 1) | (uint32_t)(lg > 1 ? lg - 1 : 0) << 8;
  }
  return SN_OK;
}

int fill_field_args(FieldArgs& a, int64_t n, const int32_t* count, const float* x,
                           const float* table, const sn_grid_desc* grid, int active_levels,
                           const sn_mlp_desc* mlp, int out_cols) {
  memset(&a, 0, sizeof(a));
  SN_REQUIRE(n >= 0, "field: n < 0");
  SN_REQUIRE(mlp != nullptr, "field: mlp descriptor is null");
  SN_TRY(make_grid_dev(grid, a.g));
  if (mlp->d_hidden != kH) {
    set_error("field: hidden width %d unsupported (kernels are built for %d)", mlp->d_hidden, kH);
    return SN_ERR_UNSUPPORTED;
  }
  SN_REQUIRE(mlp->d_in == 3 + grid->n_levels * grid->n_features,
             "field: d_in %d != 3 + levels*features", mlp->d_in);
  if (mlp->d_out < 1 || mlp->d_out > kDoutMax) {
    set_error("field: d_out %d outside 1..%d", mlp->d_out, kDoutMax);
    return SN_ERR_UNSUPPORTED;
  }
  SN_REQUIRE(out_cols >= 1 && out_cols <= mlp->d_out, "field: out_cols %d outside 1..d_out", out_cols);
  SN_REQUIRE(x && table && mlp->w0 && mlp->b0 && mlp->w1 && mlp->b1, "field: null buffer");
  a.cap = n;
  a.count = count;
  a.x = x;
  a.table = table;
  a.active = active_levels < 0 ? 0 : (active_levels > a.g.L ? a.g.L : active_levels);
  a.din = mlp->d_in;
  a.dout = mlp->d_out;
  a.out_cols = out_cols;
  a.beta = mlp->beta;
  a.thresh = mlp->threshold;
  a.w0 = mlp->w0;
  a.b0 = mlp->b0;
  a.w1 = mlp->w1;
  a.b1 = mlp->b1;
  a.status = mlp->status;
  a.table_half = (mlp->flags & SN_FIELD_TABLE_FP16) != 0;
  a.one_pass = (mlp->flags & SN_FIELD_MLP_TF32) != 0;
  a.bf16 = (mlp->flags & SN_FIELD_MLP_BF16) != 0;
  return SN_OK;
}

}  // namespace sn

using namespace sn;

extern "C" {

int sn_grid_desc_init(sn_grid_desc* d, int n_levels, int n_features, int log2_hashmap_size,
                      int base_resolution, float per_level_scale) {
  SN_REQUIRE(d != nullptr, "grid_desc_init: null descriptor");
  SN_REQUIRE(n_levels >= 1 && n_levels <= SN_MAX_LEVELS, "grid_desc_init: n_levels outside 1..%d",
             SN_MAX_LEVELS);
  SN_REQUIRE(n_features >= 1, "grid_desc_init: n_features < 1");
  SN_REQUIRE(log2_hashmap_size >= 1 && log2_hashmap_size <= 30, "grid_desc_init: bad log2 size");
  SN_REQUIRE(base_resolution >= 1, "grid_desc_init: base_resolution < 1");
  SN_REQUIRE(per_level_scale >= 1.0f, "grid_desc_init: per_level_scale < 1");
  memset(d, 0, sizeof(*d));
  d->n_levels = n_levels;
  d->n_features = n_features;
  // float32 level constants, each rounded once from a double evaluation so
  // every host (x86 or Arm libm) produces the same bits
  const float log2_pls = (float)log2((double)per_level_scale);
  uint32_t offset = 0;
  for (int l = 0; l < n_levels; ++l) {
    const float scale =
        (float)(exp2((double)l * (double)log2_pls) * (double)base_resolution - 1.0);
    const uint32_t res = (uint32_t)ceilf(scale) + 1u;
    const uint32_t max_params = 0xffffffffu / 2;
    const double dense = pow((double)res, 3.0);
    uint32_t params = dense > (double)max_params ? max_params : res * res * res;
    params = (params + 7u) / 8u * 8u;
    const uint32_t hsize = 1u << log2_hashmap_size;
    if (params > hsize) params = hsize;
    d->scales[l] = scale;
    d->resolutions[l] = res;
    d->offsets[l] = offset;
    offset += params;
  }
  d->offsets[n_levels] = offset;
  return SN_OK;
}

int sn_hashgrid_fwd(int64_t n, const float* x, const float* table, const sn_grid_desc* grid,
                    int active_levels, float* out, void* stream) {
  GridDev g;
  SN_TRY(make_grid_dev(grid, g));
  SN_REQUIRE(n >= 0, "hashgrid_fwd: n < 0");
  if (n == 0) return SN_OK;
  const int act = active_levels < 0 ? 0 : (active_levels > g.L ? g.L : active_levels);
  hashgrid_fwd_kernel<<<stride_grid(n * g.L, 256, 8), 256, 0, as_stream(stream)>>>(n, x, table, g,
                                                                                  act, out);
  return check_launch("hashgrid_fwd");
}

int sn_hashgrid_bwd(int64_t n, const float* x, const float* grad_out, const sn_grid_desc* grid,
                    int active_levels, float* grad_table, void* stream) {
  GridDev g;
  SN_TRY(make_grid_dev(grid, g));
  SN_REQUIRE(n >= 0, "hashgrid_bwd: n < 0");
  if (n == 0) return SN_OK;
  const int act = active_levels < 0 ? 0 : (active_levels > g.L ? g.L : active_levels);
  hashgrid_bwd_kernel<<<stride_grid(n * g.L, 256, 8), 256, 0, as_stream(stream)>>>(
      n, x, grad_out, g, act, grad_table);
  return check_launch("hashgrid_bwd");
}

int sn_field_fwd(int64_t n, const int32_t* count, const float* x, const float* table,
                 const sn_grid_desc* grid, int active_levels, const sn_mlp_desc* mlp, int out_cols,
                 float* out, void* stream) {
  FieldArgs a;
  SN_TRY(fill_field_args(a, n, count, x, table, grid, active_levels, mlp, out_cols));
  SN_REQUIRE(out != nullptr, "field_fwd: out is null");
  a.out = out;
  if (mlp->enc_cache) {
    SN_REQUIRE((reinterpret_cast<uintptr_t>(mlp->enc_cache) & 7u) == 0, "field_fwd: enc_cache not 8-byte aligned");
    a.enc_out = reinterpret_cast<float2*>(mlp->enc_cache);
  }
  if (n == 0) return SN_OK;
  return field_fwd_tc(a, as_stream(stream));
}

int sn_field_fwd_batch(int n_segments, const sn_field_segment* segments, int out_cols, void* stream) {
  SN_REQUIRE(segments != nullptr, "field_fwd_batch: null segments");
  SN_REQUIRE(n_segments >= 1 && n_segments <= SN_FIELD_MAX_SEGMENTS, "field_fwd_batch: %d segments (1..%d)",
             n_segments, SN_FIELD_MAX_SEGMENTS);
  FieldArgs args[SN_FIELD_MAX_SEGMENTS];
  int live = 0;
  for (int i = 0; i < n_segments; ++i) {
    const sn_field_segment& sg = segments[i];
    SN_REQUIRE(sg.out != nullptr, "field_fwd_batch: segment %d has no output", i);
    SN_TRY(fill_field_args(args[live], sg.n, nullptr, sg.x, reinterpret_cast<const float*>(sg.table), sg.grid,
                           sg.active_levels, sg.mlp, out_cols));
    SN_REQUIRE(sg.mlp->enc_cache == nullptr, "field_fwd_batch: segment %d asks for an encoding cache", i);
    args[live].out = sg.out;
    if (sg.n > 0) ++live;
  }
  if (live == 0) return SN_OK;
  return field_fwd_tc_segments(args, live, as_stream(stream));
}

static int field_bwd(int64_t n, const int32_t* count, const float* x, const float* grad_out, int out_cols,
                     const float* table, const sn_grid_desc* grid, int active_levels, const sn_mlp_desc* mlp,
                     float* grad_table, float* grad_w0, float* grad_b0, float* grad_w1, double* w1_sums,
                     float* grad_b1, float* grad_x, void* stream) {
  FieldArgs a;
  SN_TRY(fill_field_args(a, n, count, x, table, grid, active_levels, mlp, out_cols));
  if (a.bf16) {
    set_error("field_bwd: SN_FIELD_MLP_BF16 is supported by sn_field_fwd only");
    return SN_ERR_UNSUPPORTED;
  }
  SN_REQUIRE(grad_out != nullptr, "field_bwd: grad_out is null");
  a.grad_out = grad_out;
  a.grad_table = grad_table;
  a.grad_w0 = grad_w0;
  a.grad_b0 = grad_b0;
  a.grad_w1 = grad_w1;
  a.w1_sums = w1_sums;
  a.grad_x = grad_x;
  if (mlp->enc_cache) {
    SN_REQUIRE((reinterpret_cast<uintptr_t>(mlp->enc_cache) & 7u) == 0, "field_bwd: enc_cache not 8-byte aligned");
    a.enc_in = reinterpret_cast<const float2*>(mlp->enc_cache);
  }
  if (n == 0) return SN_OK;
  SN_TRY(add_bias_grad(a, grad_out, out_cols, grad_b1, as_stream(stream)));
  return field_bwd_tc(a, as_stream(stream));
}

int sn_field_bwd(int64_t n, const int32_t* count, const float* x, const float* grad_out,
                 int out_cols, const float* table, const sn_grid_desc* grid, int active_levels,
                 const sn_mlp_desc* mlp, float* grad_table, float* grad_w0, float* grad_b0,
                 float* grad_w1, float* grad_b1, float* grad_x, void* stream) {
  return field_bwd(n, count, x, grad_out, out_cols, table, grid, active_levels, mlp, grad_table, grad_w0, grad_b0,
                   grad_w1, nullptr, grad_b1, grad_x, stream);
}

int sn_field_grad_fwd(int64_t n, const int32_t* count, const float* x, const float* table,
                      const sn_grid_desc* grid, int active_levels, const sn_mlp_desc* mlp,
                      float* sdf, float* grad, void* stream) {
  FieldArgs a;
  SN_TRY(fill_field_args(a, n, count, x, table, grid, active_levels, mlp, 1));
  if (a.table_half || a.one_pass || a.bf16) {
    set_error("field_grad: SN_FIELD_* precision flags are supported by the fused field forward/backward only");
    return SN_ERR_UNSUPPORTED;
  }
  SN_REQUIRE(grad != nullptr, "field_grad_fwd: grad is null");
  if (n == 0) return SN_OK;
  return field_grad_fwd_tc(a, sdf, grad, as_stream(stream));
}

static int field_grad_bwd(int64_t n, const int32_t* count, const float* x, const float* grad_grad,
                          const float* grad_sdf, const float* table, const sn_grid_desc* grid, int active_levels,
                          const sn_mlp_desc* mlp, float* grad_table, float* grad_w0, float* grad_b0, float* grad_w1,
                          double* w1_sums, float* grad_b1, void* stream) {
  FieldArgs a;
  SN_TRY(fill_field_args(a, n, count, x, table, grid, active_levels, mlp, 1));
  if (a.table_half || a.one_pass || a.bf16) {
    set_error("field_grad: SN_FIELD_* precision flags are supported by the fused field forward/backward only");
    return SN_ERR_UNSUPPORTED;
  }
  SN_REQUIRE(grad_grad != nullptr, "field_grad_bwd: grad_grad is null");
  a.grad_table = grad_table;
  a.grad_w0 = grad_w0;
  a.grad_b0 = grad_b0;
  a.grad_w1 = grad_w1;
  a.w1_sums = w1_sums;
  if (n == 0) return SN_OK;
  SN_TRY(add_bias_grad(a, grad_sdf, 1, grad_b1, as_stream(stream)));
  return field_grad_bwd_tc(a, grad_grad, grad_sdf, as_stream(stream));
}

int sn_field_grad_bwd(int64_t n, const int32_t* count, const float* x, const float* grad_grad,
                      const float* grad_sdf, const float* table, const sn_grid_desc* grid,
                      int active_levels, const sn_mlp_desc* mlp, float* grad_table, float* grad_w0,
                      float* grad_b0, float* grad_w1, float* grad_b1, void* stream) {
  return field_grad_bwd(n, count, x, grad_grad, grad_sdf, table, grid, active_levels, mlp, grad_table, grad_w0,
                        grad_b0, grad_w1, nullptr, grad_b1, stream);
}

int sn_field_wn_fwd(int64_t n, const int32_t* count, const float* x, const float* table, const sn_grid_desc* grid,
                    int active_levels, const sn_mlp_desc* mlp, const sn_weightnorm_layer* layer0,
                    const sn_weightnorm_layer* layer1, int out_cols, float* out, void* stream) {
  SN_TRY(check_wn(mlp, layer0, layer1));
  SN_TRY(sn_weightnorm_pair_fwd(layer0, layer1, stream));
  return sn_field_fwd(n, count, x, table, grid, active_levels, mlp, out_cols, out, stream);
}

int sn_field_wn_bwd(int64_t n, const float* x, const float* grad_out, int out_cols, const float* table,
                    int64_t n_table, const sn_grid_desc* grid, int active_levels, const sn_mlp_desc* mlp,
                    const sn_weightnorm_layer* layer0, const sn_weightnorm_layer* layer1, float* grad_table,
                    float* grad_b0, float* grad_b1, float* grad_x, void* stream) {
  SN_TRY(check_wn(mlp, layer0, layer1));
  SN_TRY(begin_field_grads(*layer0, *layer1, grad_table, n_table, grad_b0, grad_b1, n, grad_out, out_cols,
                           as_stream(stream)));
  SN_TRY(field_bwd(n, nullptr, x, grad_out, out_cols, table, grid, active_levels, mlp, grad_table, layer0->grad_w,
                   grad_b0, layer1->grad_w, layer1->grad_w_sums, nullptr, grad_x, stream));
  return layer0->grad_w || layer1->grad_w ? sn_weightnorm_pair_bwd(layer0, layer1, stream) : SN_OK;
}

int sn_field_wn_grad_fwd(int64_t n, const float* x, const float* table, const sn_grid_desc* grid, int active_levels,
                         const sn_mlp_desc* mlp, const sn_weightnorm_layer* layer0, const sn_weightnorm_layer* layer1,
                         float* sdf, float* grad, void* stream) {
  SN_TRY(check_wn(mlp, layer0, layer1));
  SN_TRY(sn_weightnorm_pair_fwd(layer0, layer1, stream));
  return sn_field_grad_fwd(n, nullptr, x, table, grid, active_levels, mlp, sdf, grad, stream);
}

int sn_field_wn_grad_bwd(int64_t n, const float* x, const float* grad_grad, const float* grad_sdf, const float* table,
                         int64_t n_table, const sn_grid_desc* grid, int active_levels, const sn_mlp_desc* mlp,
                         const sn_weightnorm_layer* layer0, const sn_weightnorm_layer* layer1, float* grad_table,
                         float* grad_b0, float* grad_b1, void* stream) {
  SN_TRY(check_wn(mlp, layer0, layer1));
  SN_TRY(begin_field_grads(*layer0, *layer1, grad_table, n_table, grad_b0, grad_b1, n, grad_sdf, 1,
                           as_stream(stream)));
  SN_TRY(field_grad_bwd(n, nullptr, x, grad_grad, grad_sdf, table, grid, active_levels, mlp, grad_table,
                        layer0->grad_w, grad_b0, layer1->grad_w, layer1->grad_w_sums, nullptr, stream));
  return layer0->grad_w || layer1->grad_w ? sn_weightnorm_pair_bwd(layer0, layer1, stream) : SN_OK;
}

int sn_weightnorm_fwd(int rows, int cols, const float* v, const float* g, float* w, float* norms,
                      void* stream) {
  SN_REQUIRE(rows > 0 && cols > 0, "weightnorm_fwd: bad shape");
  WeightNormArgs a;
  a.layer[0] = a.layer[1] = sn_weightnorm_layer{rows, cols, v, g, w, norms, nullptr, nullptr, nullptr, nullptr};
  launch_chained(weightnorm_kernel<false>, dim3(div_up(rows, 4), 1), 128, 0, as_stream(stream), a);
  return check_launch("weightnorm_fwd");
}

int sn_weightnorm_bwd(int rows, int cols, const float* v, const float* g, const float* norms,
                      const float* grad_w, float* grad_v, float* grad_g, void* stream) {
  SN_REQUIRE(rows > 0 && cols > 0, "weightnorm_bwd: bad shape");
  WeightNormArgs a;
  a.layer[0] = a.layer[1] = sn_weightnorm_layer{rows, cols, v, g, nullptr, const_cast<float*>(norms),
                                                const_cast<float*>(grad_w), grad_v, grad_g, nullptr};
  launch_chained(weightnorm_kernel<true>, dim3(div_up(rows, 4), 1), 128, 0, as_stream(stream), a);
  return check_launch("weightnorm_bwd");
}

int sn_weightnorm_pair_fwd(const sn_weightnorm_layer* layer0, const sn_weightnorm_layer* layer1, void* stream) {
  WeightNormArgs a;
  SN_TRY(weightnorm_layers(layer0, layer1, false, a.layer));
  const int rows = a.layer[0].rows > a.layer[1].rows ? a.layer[0].rows : a.layer[1].rows;
  launch_chained(weightnorm_kernel<false>, dim3(div_up(rows, 4), 2), 128, 0, as_stream(stream), a);
  return check_launch("weightnorm_pair_fwd");
}

int sn_weightnorm_pair_bwd(const sn_weightnorm_layer* layer0, const sn_weightnorm_layer* layer1, void* stream) {
  WeightNormArgs a;
  SN_TRY(weightnorm_layers(layer0, layer1, true, a.layer));
  const int rows = a.layer[0].rows > a.layer[1].rows ? a.layer[0].rows : a.layer[1].rows;
  launch_chained(weightnorm_kernel<true>, dim3(div_up(rows, 4), 2), 128, 0, as_stream(stream), a);
  return check_launch("weightnorm_pair_bwd");
}

int sn_selftest_bounded_wait(uint32_t polls, int32_t* status, void* stream) {
  SN_REQUIRE(status != nullptr, "selftest_bounded_wait: status is null");
  return bounded_wait_selftest(status, polls, as_stream(stream));
}

uint32_t sn_bounded_wait_polls(void) { return bounded_wait_limit(); }

}  // extern "C"
