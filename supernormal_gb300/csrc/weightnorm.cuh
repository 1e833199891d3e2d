// Weight normalisation (torch.nn.utils.weight_norm, dim=0) of one row by one warp,
// shared by the launches that contain it.
#pragma once

#include "common.cuh"

namespace sn {

// w = g v / |v| and |v|; zero: the row of the weight gradient is cleared.
__device__ __forceinline__ void weightnorm_row(const sn_weightnorm_layer& a, int r, int lane, bool zero) {
  const float* v = a.v + (int64_t)r * a.cols;
  float s = 0.0f;
  for (int c = lane; c < a.cols; c += 32) s = fmaf(v[c], v[c], s);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  const float nrm = sqrtf(s);
  const float k = a.g[r] / nrm;
  for (int c = lane; c < a.cols; c += 32) {
    a.w[(int64_t)r * a.cols + c] = v[c] * k;
    if (zero && a.grad_w) a.grad_w[(int64_t)r * a.cols + c] = 0.0f;
  }
  if (lane == 0 && a.norms) a.norms[r] = nrm;
}

// grad_v and grad_g of a row from grad_w, or, where they are given, from its sums in
// double (then v . grad_w, which cancels, is in double too).
__device__ __forceinline__ void weightnorm_row_bwd(const sn_weightnorm_layer& a, int r, int lane) {
  const float* v = a.v + (int64_t)r * a.cols;
  float* gw = a.grad_w + (int64_t)r * a.cols;
  float s = 0.0f;
  if (a.grad_w_sums) {
    double d = 0.0;
    for (int c = lane; c < a.cols; c += 32) {
      const double w = a.grad_w_sums[(int64_t)r * a.cols + c];
      gw[c] = (float)w;   // read below by the same lane
      d += w * (double)v[c];
    }
    for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    s = (float)d;
  } else {
    for (int c = lane; c < a.cols; c += 32) s = fmaf(gw[c], v[c], s);
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  const float nrm = a.norms[r];
  const float dg = s / nrm;
  const float k = a.g[r] / nrm;
  const float m = dg / nrm;
  for (int c = lane; c < a.cols; c += 32) a.grad_v[(int64_t)r * a.cols + c] = k * (gw[c] - v[c] * m);
  if (lane == 0) a.grad_g[r] = dg;
}

// The two layers of a call, checked (adjoint: their gradients too).
inline int weightnorm_layers(const sn_weightnorm_layer* l0, const sn_weightnorm_layer* l1, bool adjoint,
                             sn_weightnorm_layer out[2]) {
  SN_REQUIRE(l0 && l1, "weightnorm: null layer");
  out[0] = *l0;
  out[1] = *l1;
  for (int i = 0; i < 2; ++i) {
    SN_REQUIRE(out[i].rows > 0 && out[i].cols > 0 && out[i].rows <= 1 << 20, "weightnorm: bad shape");
    SN_REQUIRE(out[i].v && out[i].g, "weightnorm: null weight");
    if (adjoint)
      SN_REQUIRE(out[i].norms && out[i].grad_w && out[i].grad_v && out[i].grad_g, "weightnorm: null gradient");
    else
      SN_REQUIRE(out[i].w != nullptr, "weightnorm: null output");
  }
  return SN_OK;
}

}  // namespace sn
