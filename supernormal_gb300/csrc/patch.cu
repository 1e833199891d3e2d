// Fused patch render of SuperNormal's training step (models/renderer.py:164-267):
// NeuS alpha, patch weights w = alpha * T (NA/nerfacc/cuda/csrc/render_weight.cu:87-118),
// dfd normals (models/renderer.py:187-223) or given 'ad' gradients, accumulation of
// normals and mask, and, in training mode, the losses of exp_runner.py:191-203 with
// the whole adjoint back to the field outputs.
//
// Layout: one block per patch, one warp per pixel of the patch, and the lanes of a
// warp take 32 consecutive samples of that pixel ray at a time.  Per-sample work
// (alpha, dfd, adjoints) is parallel across lanes; the transmittance product and
// the adjoint's suffix sums are warp scans with a carry between 32-sample chunks;
// dfd neighbours (same sample, adjacent pixels) are exchanged through shared
// memory.  Field-point layout: start (i, k) at i*P + k, the end of diff sample i
// at (S + slot_i)*P + k.
#include "cluster.cuh"
#include "neus_common.cuh"

#include <string.h>

namespace sn {

enum PatchMode { kFwd = 0, kBwd = 1, kTrain = 2 };

struct PatchArgs {
  int64_t n_patches;
  int H, W, P;
  const int32_t* packed;    // (n_patches, 2) over compacted samples
  const int32_t* s_count;   // device S (nullable: s_cap)
  int64_t s_cap;
  const int32_t* endp;      // (S, 2) {slot, diff}
  const float* sdf;         // field outputs, layout [S*P starts][E*P ends]
  const float* tps;         // (S, P)
  const float* tpe;         // (S, P)
  const float* ro;          // (n_patches, P, 3)
  const float* rd;          // (n_patches, P, 3)
  const float* vinv;        // (n_patches, P, 3, 3)
  const float* variance;    // device scalar
  float* alpha;             // forward outputs (nullable)
  float* weights;
  float* grads;             // (S, P, 3)
  float* comp_normal;       // (n_patches, P, 3)
  float* weight_sum;        // (n_patches, P)
  const float* g_comp;      // backward inputs
  const float* g_wsum;
  const float* g_grads;     // (S, P, 3) nullable
  const float* gt_normal;   // training inputs
  const float* gt_mask;
  const float* mask_sum;
  int loss_l1;
  float w_normal, w_eik, w_mask;
  float* d_sdf;             // backward outputs
  float* partials;          // (n_patches, 4): d_inv_s, normal, bce, eikonal
  float* carry;             // (n_patches, P)
  const float* ext_grads;   // 'ad': (S, P, 3) gradients from the field, nullable
  float* d_grads;           // 'ad': dL / d gradients
};

struct PixelRay {
  int k, r, c;
  float o[3], d[3], V[9];
};

struct Sample {
  float s0, s1, ts, te, dt, alpha, q, cdf0, cdf1;
  float g[3];
  float dxl, dxr, dyu, dyd;
  int diff, slot;
};

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ float dist3(const float* a, const float* b) {
  const float x = __fsub_rn(a[0], b[0]), y = __fsub_rn(a[1], b[1]), z = __fsub_rn(a[2], b[2]);
  return sqrtf(__fadd_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y)), __fmul_rn(z, z)));
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
}

// One pixel ray's samples: pointers to its first and 32-bit offsets from them.
struct RayView {
  const int2* endp;
  const float *sdf, *tps, *tpe;
  const float* ends;   // end value of slot 0
  int P;
  int count;           // samples of the ray (S clamps a packed table past capacity)
  int left;            // samples from the ray's first to the last of all
};
__device__ __forceinline__ RayView ray_view(const PatchArgs& a, int k, int64_t base, int64_t S, int steps) {
  RayView v;
  const int64_t o = base * a.P + k;
  v.endp = reinterpret_cast<const int2*>(a.endp) + base;
  v.sdf = a.sdf + o;
  v.tps = a.tps + o;
  v.tpe = a.tpe + o;
  v.ends = a.sdf + S * a.P + k;
  v.P = a.P;
  v.left = (int)min(max(S - base, (int64_t)0), (int64_t)0x7fffffff);
  v.count = min(steps, v.left);
  return v;
}

// What a sample reads from memory, loaded a chunk ahead of its use (its end value,
// whose address the slot gives, follows when the chunk is processed).
struct Raw {
  int2 ep;
  float s0, ts, te, next;  // next: the following start, where no other lane holds it
  bool ok;
};

__device__ __forceinline__ Raw load_raw(const RayView& v, int k, int c, int lane) {
  const int j = 32 * c + lane, o = j * v.P;
  Raw r;
  r.ok = c >= 0 && j < v.count;
  // a lane without a sample computes on values that divide plainly (no zero
  // operands): one such lane would send its warp through every division's slow path
  r.ep = make_int2(0, 0);
  r.s0 = 1.0f + (float)k;
  r.next = 0.5f;
  r.ts = 1.0f;
  r.te = 2.0f;
  if (r.ok) {
    r.ep = v.endp[j];
    r.s0 = v.sdf[o];
    r.ts = v.tps[o];
    r.te = v.tpe[o];
    if (lane == 31 || j + 1 >= v.count) r.next = j + 1 < v.left ? v.sdf[o + v.P] : r.s0;
  }
  return r;
}

// Per-sample quantities that need no neighbour pixel.
__device__ __forceinline__ void make_sample(const RayView& v, const Raw& r, float inv_s, int lane, Sample& s) {
  const float end = r.ok && r.ep.y ? v.ends[(int64_t)r.ep.x * v.P] : 0.0f;
  const float down = __shfl_down_sync(kFull, r.s0, 1);
  const bool next_ok = __shfl_down_sync(kFull, (int)r.ok, 1) != 0 && lane < 31;
  s.diff = r.ep.y;
  s.slot = r.ep.x;
  s.s0 = r.s0;
  s.s1 = r.ep.y ? end : (next_ok ? down : r.next);
  s.ts = r.ts;
  s.te = r.te;
  s.dt = __fsub_rn(s.te, s.ts);
  s.alpha = neus_alpha(s.s0, s.s1, inv_s, &s.cdf0, &s.cdf1, &s.q);
  if (!r.ok) s.alpha = 0.0f;
}

// Stages s0 and the start point in shared memory for the dfd of the other pixels.
__device__ __forceinline__ void stage_sample(const PatchArgs& a, const PixelRay& R, const Raw& r, int lane,
                                             float* sm_s0, float* sm_pos) {
  sm_s0[lane * a.P + R.k] = r.s0;
#pragma unroll
  for (int d = 0; d < 3; ++d) sm_pos[(lane * a.P + R.k) * 3 + d] = __fadd_rn(R.o[d], __fmul_rn(R.d[d], r.ts));
}

// dfd gradient (models/renderer.py:187-223) from the staged neighbours.
__device__ __forceinline__ void dfd_grad(const PatchArgs& a, const PixelRay& R, int lane,
                                         const float* sm_s0, const float* sm_pos, Sample& s) {
  const int P = a.P, W = a.W, H = a.H, k = R.k;
  const int kl = R.c > 0 ? k - 1 : k, kr = R.c < W - 1 ? k + 1 : k;
  const int ku = R.r > 0 ? k - W : k, kd = R.r < H - 1 ? k + W : k;
  const float* pos = sm_pos + (lane * P + k) * 3;
  const float sl = sm_s0[lane * P + kl], sr = sm_s0[lane * P + kr];
  const float su = sm_s0[lane * P + ku], sd = sm_s0[lane * P + kd];
  s.dxl = R.c > 0 ? dist3(pos, sm_pos + (lane * P + kl) * 3) : 0.0f;
  s.dxr = R.c < W - 1 ? dist3(sm_pos + (lane * P + kr) * 3, pos) : 0.0f;
  s.dyu = R.r > 0 ? dist3(pos, sm_pos + (lane * P + ku) * 3) : 0.0f;
  s.dyd = R.r < H - 1 ? dist3(sm_pos + (lane * P + kd) * 3, pos) : 0.0f;
  float proj[3];
  proj[0] = __fdiv_rn(__fsub_rn(s.s1, s.s0), s.dt);
  if (R.c == 0)
    proj[1] = __fdiv_rn(__fsub_rn(sr, s.s0), s.dxr);
  else if (R.c == W - 1)
    proj[1] = __fdiv_rn(__fsub_rn(s.s0, sl), s.dxl);
  else
    proj[1] = __fdiv_rn(__fsub_rn(sr, sl), __fadd_rn(s.dxl, s.dxr));
  if (R.r == 0)
    proj[2] = __fdiv_rn(__fsub_rn(sd, s.s0), s.dyd);
  else if (R.r == H - 1)
    proj[2] = __fdiv_rn(__fsub_rn(s.s0, su), s.dyu);
  else
    proj[2] = __fdiv_rn(__fsub_rn(sd, su), __fadd_rn(s.dyu, s.dyd));
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    float v = __fmul_rn(R.V[3 * e + 0], proj[0]);
    v = __fadd_rn(v, __fmul_rn(R.V[3 * e + 1], proj[1]));
    v = __fadd_rn(v, __fmul_rn(R.V[3 * e + 2], proj[2]));
    s.g[e] = v;
  }
}

// The sample's gradient: the given one, or dfd from the staged neighbours (one
// block barrier; buf alternates, so the next chunk is staged beside this one).
__device__ __forceinline__ void sample_gradient(const PatchArgs& a, const PixelRay& R, int64_t i, const Raw& r,
                                                int lane, float* sm, int& buf, Sample& s) {
  if (a.ext_grads) {
#pragma unroll
    for (int e = 0; e < 3; ++e) s.g[e] = r.ok ? a.ext_grads[(i * a.P + R.k) * 3 + e] : 0.0f;
    s.dxl = s.dxr = s.dyu = s.dyd = 0.0f;
    return;
  }
  float* sm_s0 = sm + buf * 128 * a.P;
  float* sm_pos = sm_s0 + 32 * a.P;
  stage_sample(a, R, r, lane, sm_s0, sm_pos);
  __syncthreads();
  buf ^= 1;
  dfd_grad(a, R, lane, sm_s0, sm_pos, s);
  if (!r.ok) s.g[0] = s.g[1] = s.g[2] = 0.0f;
}

// Transmittance T_j = prod_{i<j} (1 - alpha_i) along the pixel ray: the
// exclusive product over the lanes of 1 - alpha (formed exactly as a
// double-float), times the running carry of the earlier chunks (which
// advances).  Double-float throughout, so T keeps ~2^-44 relative accuracy
// over a thousand samples where a float32 running product drifts by ~j ulp.
__device__ __forceinline__ ff transmittance(float alpha, bool ok, ff& carry, int lane) {
  ff incl = ok ? two_sum(1.0f, -alpha) : ff{1.0f, 0.0f};
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const ff y = shfl_up_ff(incl, o);
    if (lane >= o) incl = ff_mul(y, incl);
  }
  ff excl = shfl_up_ff(incl, 1);
  if (lane == 0) excl = ff{1.0f, 0.0f};
  const ff T = ff_mul(carry, excl);
  carry = ff_mul(carry, shfl_ff(incl, 31));
  return T;
}

// d loss / d w_j of one sample: the rendered-normal gradient along the
// sample's gradient plus the weight-sum gradient (one expression for every
// pass, so the passes see the same rounded values).
__device__ __forceinline__ float weight_grad(const float gc[3], float gws, const float g[3]) {
  return __fadd_rn(__fmaf_rn(gc[2], g[2], __fmaf_rn(gc[1], g[1], __fmul_rn(gc[0], g[0]))), gws);
}

// Chunks whose transmittance carry the forward walk keeps for the adjoint (more
// chunks: every 2nd, 3rd, ... is kept and the ones between are walked again).
constexpr int kKeptCarries = 40;
constexpr size_t patch_smem(int P) { return (size_t)P * (384 * sizeof(float) + kKeptCarries * sizeof(ff)); }

// Two walks over a ray's chunks of 32 samples: front to back for the rendered
// values, then, for the adjoint, back to front with the kept transmittances, so
// the suffix sums it needs run along with it.  A block lasts as long as its
// patch's longest ray is (few patches see the surface, so the launch is one
// wave and its time is its longest block's): what counts is the chain per chunk,
// hence the loads a chunk ahead and one barrier per exchange.  With a third walk
// for the total of the weight gradients and two barriers per exchange, 2,048
// patches (38 kept samples a centre ray) took 130 us; now 97 us, and 512 patches
// 80 -> 59 us.
// 3x3 patches (288 threads): at least three blocks per SM (72 registers);
// unbounded, the kernel takes 96 registers and only two blocks fit.
template <int MODE, int MAXT>
__global__ void __launch_bounds__(MAXT, MAXT == 288 ? 3 : 1) patch_block_kernel(PatchArgs a) {
  chained();
  extern __shared__ float sm[];
  const int P = a.P;
  // [2][32][P] starts and [32][P][3] points of two chunks, then
  float* sm_x = sm + 256 * P;                                // [32][P][4] dfd adjoint exchange
  ff* sm_carry = reinterpret_cast<ff*>(sm + 384 * P);        // [kKeptCarries][P]
  __shared__ float red[32][4];
  const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t p = blockIdx.x;
  PixelRay R;
  R.k = k;
  R.r = k / a.W;
  R.c = k - R.r * a.W;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    R.o[d] = a.ro[(p * P + k) * 3 + d];
    R.d[d] = a.rd[(p * P + k) * 3 + d];
  }
#pragma unroll
  for (int e = 0; e < 9; ++e) R.V[e] = a.vinv[(p * P + k) * 9 + e];
  const int64_t S = a.s_count ? min((int64_t)*a.s_count, a.s_cap) : a.s_cap;
  const int64_t base = a.packed[2 * p];
  const int steps = a.packed[2 * p + 1];
  const int chunks = (steps + 31) >> 5;
  const RayView view = ray_view(a, k, base, S, steps);
  const int kept_every = (chunks + kKeptCarries - 1) / kKeptCarries;
  const float inv_s = inv_s_from(a.variance);
  if (MODE != kFwd && lane == 0) a.carry[p * P + k] = 0.0f;

  // ---------------- forward ----------------
  int buf = 0;
  ff Tc{1.0f, 0.0f};
  float cp0 = 0.0f, cp1 = 0.0f, cp2 = 0.0f, ws = 0.0f, eik = 0.0f;
  Raw ahead = load_raw(view, k, 0, lane);
  for (int c = 0; c < chunks; ++c) {
    const Raw raw = ahead;
    ahead = load_raw(view, k, c + 1, lane);
    const int64_t i = base + 32 * c + lane;
    Sample s;
    make_sample(view, raw, inv_s, lane, s);
    if (MODE != kBwd) sample_gradient(a, R, i, raw, lane, sm, buf, s);
    if (MODE != kFwd && lane == 0 && c % kept_every == 0) sm_carry[(c / kept_every) * P + k] = Tc;
    const ff Tf = transmittance(s.alpha, raw.ok, Tc, lane);
    if (MODE == kBwd) continue;
    const float w = raw.ok ? __fmul_rn(s.alpha, ff_val(Tf)) : 0.0f;
    ws = __fadd_rn(ws, w);
    cp0 = __fadd_rn(cp0, __fmul_rn(w, s.g[0]));
    cp1 = __fadd_rn(cp1, __fmul_rn(w, s.g[1]));
    cp2 = __fadd_rn(cp2, __fmul_rn(w, s.g[2]));
    if (MODE == kFwd && raw.ok) {
      if (a.alpha) a.alpha[i * P + k] = s.alpha;
      if (a.weights) a.weights[i * P + k] = w;
      if (a.grads) {
#pragma unroll
        for (int e = 0; e < 3; ++e) a.grads[(i * P + k) * 3 + e] = s.g[e];
      }
    }
    if (MODE == kTrain && raw.ok) {
      const float nr = sqrtf(s.g[0] * s.g[0] + s.g[1] * s.g[1] + s.g[2] * s.g[2]);
      eik += (nr - 1.0f) * (nr - 1.0f);
    }
  }
  if (MODE != kBwd) {
    ws = warp_sum(ws);
    cp0 = warp_sum(cp0);
    cp1 = warp_sum(cp1);
    cp2 = warp_sum(cp2);
    if (MODE == kFwd) {
      if (lane == 0) {
        a.comp_normal[(p * P + k) * 3 + 0] = cp0;
        a.comp_normal[(p * P + k) * 3 + 1] = cp1;
        a.comp_normal[(p * P + k) * 3 + 2] = cp2;
        a.weight_sum[p * P + k] = ws;
      }
      return;
    }
  }

  // ---------------- output gradients ----------------
  float gc[3], gws, eik_scale = 0.0f;
  if (MODE == kTrain) {
    const float m = a.gt_mask[p * P + k];
    const float msum = *a.mask_sum;
    const float cp[3] = {cp0, cp1, cp2};
    float nl = 0.0f;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      const float err = __fmul_rn(__fsub_rn(cp[e], a.gt_normal[(p * P + k) * 3 + e]), m);
      if (a.loss_l1) {
        nl += fabsf(err);
        const float sg = err > 0.0f ? 1.0f : (err < 0.0f ? -1.0f : 0.0f);
        gc[e] = a.w_normal * sg * m / msum;
      } else {
        nl += err * err;
        gc[e] = a.w_normal * 2.0f * err * m / msum;
      }
    }
    const float npix = (float)(a.n_patches * P);
    const float cl = fminf(fmaxf(ws, 1e-5f), 1.0f - 1e-5f);
    const float bce = -(m * fmaxf(logf(cl), -100.0f) + (1.0f - m) * fmaxf(logf(1.0f - cl), -100.0f));
    const bool pass = ws >= 1e-5f && ws <= 1.0f - 1e-5f;
    gws = pass ? a.w_mask * (cl - m) / fmaxf((1.0f - cl) * cl, 1e-12f) / npix : 0.0f;
    eik_scale = a.w_eik * 2.0f / (float)(S * P);
    eik = warp_sum(eik);
    if (lane == 0) {
      red[k][1] = nl;
      red[k][2] = bce;
      red[k][3] = eik;
    }
  } else {
#pragma unroll
    for (int e = 0; e < 3; ++e) gc[e] = a.g_comp[(p * P + k) * 3 + e];
    gws = a.g_wsum[p * P + k];
  }

  // ---------------- adjoint per sample, back to front ----------------
  const int W = a.W, H = a.H;
  const int kl = R.c > 0 ? k - 1 : k, kr = R.c < W - 1 ? k + 1 : k;
  const int ku = R.r > 0 ? k - W : k, kd = R.r < H - 1 ? k + W : k;
  float d_inv = 0.0f;
  ff behind{0.0f, 0.0f};   // sum of g_i w_i over the later chunks
  float held = 0.0f;       // lane 0: the later chunk's first start adjoint, before what this one adds
  __syncwarp();            // lane 0's kept carries
  ahead = load_raw(view, k, chunks - 1, lane);
  for (int c = chunks - 1; c >= 0; --c) {
    const int j = 32 * c + lane;
    const int64_t i = base + j;
    const Raw raw = ahead;
    const bool ok = raw.ok;
    ahead = load_raw(view, k, c - 1, lane);
    Sample s;
    make_sample(view, raw, inv_s, lane, s);
    sample_gradient(a, R, i, raw, lane, sm, buf, s);
    Tc = sm_carry[(c / kept_every) * P + k];
    for (int b = c - c % kept_every; b < c; ++b) {
      Sample e;
      make_sample(view, load_raw(view, k, b, lane), inv_s, lane, e);
      transmittance(e.alpha, 32 * b + lane < view.count, Tc, lane);
    }
    const ff Tf = transmittance(s.alpha, ok, Tc, lane);
    const float T = ff_val(Tf);
    const float w = ok ? __fmul_rn(s.alpha, T) : 0.0f;
    const float gw = ok ? weight_grad(gc, gws, s.g) : 0.0f;
    // accum_j = sum_{i >= j} g_i w_i (NA/nerfacc/cuda/csrc/render_weight.cu:325-337)
    // = this chunk's suffix scan + the chunks behind, in double-float.  The
    // terms g_i alpha_i T_i are double-float products: with T carried as
    // prod (1 - alpha) from exact differences, T_j - sum_{i >= j} alpha_i T_i
    // telescopes to the transmittance past the ray's end, so the numerator
    // g_j T_j - accum_j keeps its digits when that remainder is small (an
    // opaque ray), where float32 terms would leave rounding noise of order
    // eps * g_j T_j.  Summed from the back, a suffix has no larger sum to be
    // the difference of.
    ff accum = ok ? ff_mul(ff{gw, 0.0f}, ff_mul(Tf, ff{s.alpha, 0.0f})) : ff{0.0f, 0.0f};
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const ff y = shfl_down_ff(accum, o);
      if (lane + o < 32) accum = ff_add(y, accum);
    }
    accum = ff_add(behind, accum);
    behind = shfl_ff(accum, 0);
    const float num = ff_val(ff_add(ff_mul(ff{gw, 0.0f}, Tf), ff_neg(accum)));
    const float dalpha = __fdiv_rn(ok ? num : 1.0f, fmaxf(__fsub_rn(1.0f, s.alpha), 1e-10f));
    // alpha = clip(q): sigmoid terms (1 divided in place of a clipped sample's 0:
    // zero operands leave the division's fast path).  d q / d cdf0 could be taken as
    // cdf1/ce^2, without the difference, but sums of these adjoints over the samples
    // cancel to a few ulp of them, and there the order of rounding shows.
    const float dq = (ok && s.q >= 0.0f && s.q <= 1.0f) ? dalpha : 0.0f;
    const float ce = s.cdf0 + 1e-5f;
    const float through = dq != 0.0f ? 1.0f : 0.0f;
    const float dp = __fdiv_rn(dq != 0.0f ? dq : 1.0f, ce) * through;
    const float dd = dq != 0.0f ? dq * (s.cdf0 - s.cdf1 + 1e-5f) : 1.0f;
    const float dc = dp - __fdiv_rn(dd, ce * ce) * through;
    const float dn = -dp;
    const float dx0 = dc * s.cdf0 * (1.0f - s.cdf0);
    const float dx1 = dn * s.cdf1 * (1.0f - s.cdf1);
    float ds0 = dx0 * inv_s, ds1 = dx1 * inv_s;
    d_inv += dx0 * s.s0 + dx1 * s.s1;
    // gradient adjoint: accumulation + eikonal (+ caller's)
    float dg[3];
#pragma unroll
    for (int e = 0; e < 3; ++e) dg[e] = gc[e] * w;
    if (MODE == kTrain) {
      const float nr = sqrtf(s.g[0] * s.g[0] + s.g[1] * s.g[1] + s.g[2] * s.g[2]);
      if (ok && nr > 0.0f) {
        const float kk = eik_scale * (nr - 1.0f) / nr;
#pragma unroll
        for (int e = 0; e < 3; ++e) dg[e] += kk * s.g[e];
      }
    } else if (a.g_grads && ok) {
#pragma unroll
      for (int e = 0; e < 3; ++e) dg[e] += a.g_grads[(i * P + k) * 3 + e];
    }
    if (a.ext_grads) {
      if (ok) {
#pragma unroll
        for (int e = 0; e < 3; ++e) a.d_grads[(i * P + k) * 3 + e] = dg[e];
      }
    } else {
      float dpj[3];
#pragma unroll
      for (int b = 0; b < 3; ++b) dpj[b] = R.V[b] * dg[0] + R.V[3 + b] * dg[1] + R.V[6 + b] * dg[2];
      const float gt = ok ? dpj[0] / s.dt : 0.0f;
      ds1 += gt;
      ds0 -= gt;
      float to_l = 0.0f, to_r = 0.0f, to_u = 0.0f, to_d = 0.0f;
      if (ok) {
        if (R.c == 0) {
          const float g = dpj[1] / s.dxr;
          to_r += g;
          ds0 -= g;
        } else if (R.c == W - 1) {
          const float g = dpj[1] / s.dxl;
          ds0 += g;
          to_l -= g;
        } else {
          const float g = dpj[1] / (s.dxl + s.dxr);
          to_r += g;
          to_l -= g;
        }
        if (R.r == 0) {
          const float g = dpj[2] / s.dyd;
          to_d += g;
          ds0 -= g;
        } else if (R.r == H - 1) {
          const float g = dpj[2] / s.dyu;
          ds0 += g;
          to_u -= g;
        } else {
          const float g = dpj[2] / (s.dyu + s.dyd);
          to_d += g;
          to_u -= g;
        }
      }
      float* x = sm_x + (lane * P + k) * 4;
      x[0] = to_l;
      x[1] = to_r;
      x[2] = to_u;
      x[3] = to_d;
      __syncthreads();  // (the next write of sm_x is behind the next chunk's barrier)
      if (R.c > 0) ds0 += sm_x[(lane * P + kl) * 4 + 1];      // left neighbour's "to right"
      if (R.c < W - 1) ds0 += sm_x[(lane * P + kr) * 4 + 0];  // right neighbour's "to left"
      if (R.r > 0) ds0 += sm_x[(lane * P + ku) * 4 + 3];      // upper neighbour's "to down"
      if (R.r < H - 1) ds0 += sm_x[(lane * P + kd) * 4 + 2];  // lower neighbour's "to up"
    }
    // route the end adjoint: its own end point, the next start of this ray, or
    // (after the patch's last sample) the next patch's first start via `carry`
    const bool to_next = ok && !s.diff && (j + 1 < steps);
    const float routed = to_next ? ds1 : 0.0f;
    const float prev = __shfl_up_sync(kFull, routed, 1);
    const float last = __shfl_sync(kFull, routed, 31);
    if (lane == 0 && c + 1 < chunks && j + 32 < view.count) a.d_sdf[(i + 32) * P + k] = held + last;
    if (ok) {
      if (lane > 0) ds0 += prev;
      if (s.diff) {
        a.d_sdf[(S + s.slot) * P + k] = ds1;
      } else if (j + 1 == steps) {
        if (i + 1 < S)
          a.carry[p * P + k] = ds1;
        else
          ds0 += ds1;  // the last sample compares with itself
      }
      if (lane > 0 || c == 0)
        a.d_sdf[i * P + k] = ds0;
      else
        held = ds0;
    }
  }
  d_inv = warp_sum(d_inv);
  if (lane == 0) red[k][0] = d_inv;
  __syncthreads();
  if (threadIdx.x == 0) {
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    for (int q = 0; q < P; ++q) {
      acc[0] += red[q][0];
      if (MODE == kTrain) {
        acc[1] += red[q][1];
        acc[2] += red[q][2];
        acc[3] += red[q][3];
      }
    }
    a.partials[4 * p + 0] = acc[0];
    if (MODE == kTrain) {
      a.partials[4 * p + 1] = acc[1];
      a.partials[4 * p + 2] = acc[2];
      a.partials[4 * p + 3] = acc[3];
    }
  }
}

// Adds each patch's carried end adjoint to the start of the sample after its
// last one (only when that end was not evaluated separately).
struct Fixup {
  int64_t n_patches, s_cap;
  int P;
  const int32_t *packed, *s_count, *endp;
  const float* carry;
  float* d_sdf;
};
__device__ __forceinline__ void carry_fixup(const Fixup& a, int64_t first, int64_t step) {
  const int64_t S = a.s_count ? min((int64_t)*a.s_count, a.s_cap) : a.s_cap;
  for (int64_t t = first; t < a.n_patches * a.P; t += step) {
    const int64_t p = (t >> 32) ? t / a.P : (int64_t)((uint32_t)t / (uint32_t)a.P);
    const int k = (int)(t - p * a.P);
    const int steps = a.packed[2 * p + 1];
    if (steps == 0) continue;
    const int64_t last = (int64_t)a.packed[2 * p] + steps - 1;
    if (last + 1 >= S || a.endp[2 * last + 1]) continue;
    a.d_sdf[(last + 1) * a.P + k] += a.carry[t];
  }
}
__global__ void carry_fixup_kernel(Fixup a) {
  carry_fixup(a, blockIdx.x * (int64_t)blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x);
}

// Sums per-patch partials: grad_variance += d loss/d variance and
// out = {d/d variance, normal, bce, eikonal, total} (exp_runner.py:191-203).  The
// sums are in double, whose units do two operations a cycle and SM: one block spent
// 10 us on 2,048 patches (now 4.8 with the carries).  So a cluster of eight blocks
// sums, each warp's lanes take one sum each after two exchanges, and the first block
// adds the eight parts.
struct Finalize {
  int64_t n_patches, s_cap;
  int P;
  const float* partials;
  const int32_t* s_count;
  const float *variance, *mask_sum;
  float w_normal, w_eik, w_mask;
  float *out, *grad_variance;
};
constexpr int kFinishThreads = 256, kFinishCluster = 8;
// Block `part` of the eight of its cluster; every thread takes part and has
// arrived at the cluster's barrier once.
__device__ __forceinline__ void finalize_part(const Finalize& a, uint32_t part) {
  __shared__ double red[4][kFinishThreads / 32];
  __shared__ double parts[4][kFinishCluster];   // of the first block
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (int64_t p = part * kFinishThreads + threadIdx.x; p < a.n_patches; p += kFinishCluster * kFinishThreads) {
    float v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = a.partials[4 * p + q];
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[q] += (double)v[q];
  }
  // sum q = lane >> 3 of the warp's 32 values to the eight lanes of its group
  const bool hi = lane & 16, mid = lane & 8;
  const double a0 = (hi ? acc[2] : acc[0]) + __shfl_xor_sync(kFull, hi ? acc[0] : acc[2], 16);
  const double a1 = (hi ? acc[3] : acc[1]) + __shfl_xor_sync(kFull, hi ? acc[1] : acc[3], 16);
  double v = (mid ? a1 : a0) + __shfl_xor_sync(kFull, mid ? a0 : a1, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  if ((lane & 7) == 0) red[lane >> 3][warp] = v;
  __syncthreads();
  static_assert(kFinishThreads == 256 && kFinishCluster == 8, "eight warps and eight blocks to a sum");
  cluster_wait();   // the first block runs: its shared memory may be stored to
  if (warp == 0) {   // lane group q: the sum of the warps' parts of sum q
    v = red[lane >> 3][lane & 7];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    if ((lane & 7) == 0) st_cluster(&parts[lane >> 3][part], 0, v);
  }
  cluster_arrive();
  cluster_wait();
  if (part != 0 || warp != 0) return;
  v = parts[lane >> 3][lane & 7];
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  const double s[4] = {__shfl_sync(kFull, v, 0), __shfl_sync(kFull, v, 8), __shfl_sync(kFull, v, 16),
                       __shfl_sync(kFull, v, 24)};
  if (lane == 0) {
    const float ev = expf(__fmul_rn(*a.variance, 10.0f));
    const bool pass = ev >= 1e-6f && ev <= 1e6f;
    const float dvar = pass ? (float)s[0] * ev * 10.0f : 0.0f;
    if (a.grad_variance) *a.grad_variance += dvar;
    if (a.out) {
      const int64_t S = a.s_count ? min((int64_t)*a.s_count, a.s_cap) : a.s_cap;
      const float nl = a.mask_sum ? (float)s[1] / *a.mask_sum : 0.0f;
      const float bce = (float)(s[2] / (double)(a.n_patches * a.P));
      const float eik = S > 0 ? (float)(s[3] / (double)(S * a.P)) : 0.0f;
      a.out[0] = dvar;
      a.out[1] = nl;
      a.out[2] = bce;
      a.out[3] = eik;
      a.out[4] = a.w_normal * nl + a.w_mask * bce + a.w_eik * eik;
    }
  }
}

// Both in one launch: the first cluster sums, the others (if any) carry.
__global__ void __cluster_dims__(kFinishCluster, 1, 1) __launch_bounds__(kFinishThreads)
patch_finish_kernel(const __grid_constant__ Fixup f, const __grid_constant__ Finalize a) {
  chained();
  if (blockIdx.x < kFinishCluster) {
    cluster_arrive();   // waited for behind the loads
    finalize_part(a, cluster_rank());
  } else {
    carry_fixup(f, (blockIdx.x - kFinishCluster) * (int64_t)kFinishThreads + threadIdx.x,
                (gridDim.x - kFinishCluster) * (int64_t)kFinishThreads);
  }
}

static int patch_common(PatchArgs& a, int64_t n_patches, int patch_h, int patch_w,
                        const int32_t* packed, const int32_t* s_count, int64_t s_cap,
                        const int32_t* end_packed, const float* sdf, const float* tps,
                        const float* tpe, const float* rays_o, const float* rays_d,
                        const float* vinv, const float* variance) {
  memset(&a, 0, sizeof(a));
  SN_REQUIRE(n_patches >= 0 && s_cap >= 0, "patch_render: negative size");
  SN_REQUIRE(n_patches < (int64_t)1 << 31, "patch_render: too many patches");
  SN_REQUIRE(patch_h >= 3 && patch_w >= 3 && patch_h * patch_w <= 32,
             "patch_render: patch must be at least 3x3 and at most 32 pixels (got %dx%d)", patch_h,
             patch_w);
  SN_REQUIRE(packed && end_packed && sdf && tps && tpe && rays_o && rays_d && vinv && variance,
             "patch_render: null input");
  a.n_patches = n_patches;
  a.H = patch_h;
  a.W = patch_w;
  a.P = patch_h * patch_w;
  a.packed = packed;
  a.s_count = s_count;
  a.s_cap = s_cap;
  a.endp = end_packed;
  a.sdf = sdf;
  a.tps = tps;
  a.tpe = tpe;
  a.ro = rays_o;
  a.rd = rays_d;
  a.vinv = vinv;
  a.variance = variance;
  return SN_OK;
}

template <int MODE>
static int launch_patch(const PatchArgs& a, cudaStream_t st, const char* what) {
  if (a.n_patches == 0) return SN_OK;
  const size_t smem = patch_smem(a.P);
  const unsigned threads = 32 * a.P;
  // register budget follows the block size (3x3 patches: 72, three blocks per SM)
  const auto fn = a.P <= 9    ? patch_block_kernel<MODE, 288>
                  : a.P <= 16 ? patch_block_kernel<MODE, 512>
                              : patch_block_kernel<MODE, 1024>;
  if (smem + 1024 > 48 * 1024) SN_TRY(ensure_smem_limit(reinterpret_cast<const void*>(fn), patch_smem(32), what));
  launch_chained(fn, (unsigned)a.n_patches, threads, smem, st, a);
  return check_launch(what);
}

}  // namespace sn

using namespace sn;

extern "C" {

int sn_patch_render_fwd(int64_t n_patches, int patch_h, int patch_w, const int32_t* packed_info,
                        const int32_t* s_count, int64_t s_cap, const int32_t* end_packed,
                        const float* sdf, const float* t_pix_starts, const float* t_pix_ends,
                        const float* rays_o, const float* rays_d, const float* v_inverse,
                        const float* variance, float* alpha, float* weights, float* gradients,
                        float* comp_normal, float* weight_sum, const float* ext_gradients,
                        void* stream) {
  PatchArgs a;
  SN_TRY(patch_common(a, n_patches, patch_h, patch_w, packed_info, s_count, s_cap, end_packed, sdf,
                      t_pix_starts, t_pix_ends, rays_o, rays_d, v_inverse, variance));
  SN_REQUIRE(comp_normal && weight_sum, "patch_render_fwd: null output");
  a.ext_grads = ext_gradients;
  a.alpha = alpha;
  a.weights = weights;
  a.grads = gradients;
  a.comp_normal = comp_normal;
  a.weight_sum = weight_sum;
  return launch_patch<kFwd>(a, as_stream(stream), "patch_render_fwd");
}

int sn_patch_render_bwd(int64_t n_patches, int patch_h, int patch_w, const int32_t* packed_info,
                        const int32_t* s_count, int64_t s_cap, const int32_t* end_packed,
                        const float* sdf, const float* t_pix_starts, const float* t_pix_ends,
                        const float* rays_o, const float* rays_d, const float* v_inverse,
                        const float* variance, const float* grad_comp_normal,
                        const float* grad_weight_sum, const float* grad_gradients, float* d_sdf,
                        float* partials, float* carry, const float* ext_gradients,
                        float* d_gradients, void* stream) {
  PatchArgs a;
  SN_TRY(patch_common(a, n_patches, patch_h, patch_w, packed_info, s_count, s_cap, end_packed, sdf,
                      t_pix_starts, t_pix_ends, rays_o, rays_d, v_inverse, variance));
  SN_REQUIRE(grad_comp_normal && grad_weight_sum && d_sdf && partials && carry,
             "patch_render_bwd: null buffer");
  SN_REQUIRE(ext_gradients == nullptr || d_gradients != nullptr,
             "patch_render_bwd: d_gradients required with ext_gradients");
  a.ext_grads = ext_gradients;
  a.d_grads = d_gradients;
  a.carry = carry;
  a.g_comp = grad_comp_normal;
  a.g_wsum = grad_weight_sum;
  a.g_grads = grad_gradients;
  a.d_sdf = d_sdf;
  a.partials = partials;
  return launch_patch<kBwd>(a, as_stream(stream), "patch_render_bwd");
}

int sn_patch_render_train(int64_t n_patches, int patch_h, int patch_w, const int32_t* packed_info,
                          const int32_t* s_count, int64_t s_cap, const int32_t* end_packed,
                          const float* sdf, const float* t_pix_starts, const float* t_pix_ends,
                          const float* rays_o, const float* rays_d, const float* v_inverse,
                          const float* variance, const float* gt_normal, const float* gt_mask,
                          const float* mask_sum, int loss_l1, float w_normal, float w_eikonal,
                          float w_mask, float* d_sdf, float* partials, float* carry,
                          const float* ext_gradients, float* d_gradients, void* stream) {
  PatchArgs a;
  SN_TRY(patch_common(a, n_patches, patch_h, patch_w, packed_info, s_count, s_cap, end_packed, sdf,
                      t_pix_starts, t_pix_ends, rays_o, rays_d, v_inverse, variance));
  SN_REQUIRE(gt_normal && gt_mask && mask_sum && d_sdf && partials && carry,
             "patch_render_train: null buffer");
  SN_REQUIRE(ext_gradients == nullptr || d_gradients != nullptr,
             "patch_render_train: d_gradients required with ext_gradients");
  a.ext_grads = ext_gradients;
  a.d_grads = d_gradients;
  a.carry = carry;
  a.gt_normal = gt_normal;
  a.gt_mask = gt_mask;
  a.mask_sum = mask_sum;
  a.loss_l1 = loss_l1;
  a.w_normal = w_normal;
  a.w_eik = w_eikonal;
  a.w_mask = w_mask;
  a.d_sdf = d_sdf;
  a.partials = partials;
  return launch_patch<kTrain>(a, as_stream(stream), "patch_render_train");
}

int sn_patch_carry_fixup(int64_t n_patches, int patch_size, const int32_t* packed_info,
                         const int32_t* s_count, int64_t s_cap, const int32_t* end_packed,
                         const float* carry, float* d_sdf, void* stream) {
  SN_REQUIRE(n_patches >= 0 && patch_size >= 1, "patch_carry_fixup: bad sizes");
  if (n_patches == 0) return SN_OK;
  carry_fixup_kernel<<<stride_grid(n_patches * patch_size, 256, 8), 256, 0, as_stream(stream)>>>(
      Fixup{n_patches, s_cap, patch_size, packed_info, s_count, end_packed, carry, d_sdf});
  return check_launch("patch_carry_fixup");
}

int sn_patch_finalize(int64_t n_patches, int patch_size, const float* partials,
                      const int32_t* s_count, int64_t s_cap, const float* variance,
                      const float* mask_sum, float w_normal, float w_eikonal, float w_mask,
                      float* out, float* grad_variance, void* stream) {
  SN_REQUIRE(n_patches >= 0 && patch_size >= 1, "patch_finalize: bad sizes");
  SN_REQUIRE(partials && variance, "patch_finalize: null buffer");
  launch_chained(patch_finish_kernel, kFinishCluster, kFinishThreads, 0, as_stream(stream), Fixup{},
      Finalize{n_patches, s_cap, patch_size, partials, s_count, variance, mask_sum, w_normal, w_eikonal, w_mask,
      out, grad_variance});
  return check_launch("patch_finalize");
}

int sn_patch_finish(int64_t n_patches, int patch_size, const int32_t* packed_info, const int32_t* s_count,
                    int64_t s_cap, const int32_t* end_packed, const float* carry, float* d_sdf,
                    const float* partials, const float* variance, const float* mask_sum, float w_normal,
                    float w_eikonal, float w_mask, float* out, float* grad_variance, void* stream) {
  SN_REQUIRE(n_patches >= 0 && patch_size >= 1 && s_cap >= 0, "patch_finish: bad sizes");
  SN_REQUIRE(variance != nullptr, "patch_finish: null variance");
  SN_REQUIRE(n_patches == 0 || (packed_info && end_packed && carry && d_sdf && partials),
             "patch_finish: null buffer");
  const unsigned blocks = stride_grid(n_patches > 0 ? n_patches * patch_size : 1, kFinishThreads, 4);
  launch_chained(patch_finish_kernel,
      kFinishCluster + (blocks + kFinishCluster - 1) / kFinishCluster * kFinishCluster, kFinishThreads, 0,
      as_stream(stream), Fixup{n_patches, s_cap, patch_size, packed_info, s_count, end_packed, carry, d_sdf},
      Finalize{n_patches, s_cap, patch_size, partials, s_count, variance, mask_sum, w_normal, w_eikonal, w_mask,
      out, grad_variance});
  return check_launch("patch_finish");
}

}  // extern "C"
