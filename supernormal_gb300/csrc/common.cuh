// Shared device/host helpers for the supernormal_gb300 CUDA library.
//
// Every exported entry point is `extern "C"`, takes raw device pointers,
// element counts and a `cudaStream_t` (passed as `void*`), writes into
// caller-allocated buffers and returns an `SN_*` status code.  A failing
// status leaves a human-readable message retrievable with sn_last_error().
#pragma once

#include <utility>

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <stdarg.h>

#include "../../include/supernormal_gb300.h"

namespace sn {

// ---------------------------------------------------------------------------
// error reporting
// ---------------------------------------------------------------------------
void set_error(const char* fmt, ...);
void count_launches(int k);

// Records k kernel launches (for the launch counter) and checks for errors.
inline int check_launch(const char* what, int k = 1) {
  count_launches(k);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error("%s: CUDA launch failed: %s", what, cudaGetErrorString(e));
    return SN_ERR_CUDA;
  }
  return SN_OK;
}

// Chained launches (programmatic dependent launch) for the kernels of an iteration.
// Such a kernel is put on the SMs while its predecessor in the stream still runs
// and calls chained() before anything else: it lets its own successor come, then
// waits for the predecessor's end and its writes.  Every kernel launched so does
// that, so an end reaches down the whole chain; a kernel launched plainly waits for
// all before it as ever.  Twenty launches follow one another in an iteration, most
// of them 2-5 us, and the gap before each is now shorter: 256 patches 155 -> 151 us
// an iteration, 512 with a 2^21 table 602 -> 587, 2,048 746 -> 735 (each against the
// same earlier version on one machine).  A kernel that allocates tensor memory does so
// after the wait and lets its successor come only then: no CTA that waits for another
// grid holds any.
template <typename... P, typename... A>
inline void launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);  // check_launch reads the error
}
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chained() {
  chain_release();
  chain_wait();
}

#define SN_REQUIRE(cond, ...)          \
  do {                                 \
    if (!(cond)) {                     \
      ::sn::set_error(__VA_ARGS__);    \
      return SN_ERR_INVALID;           \
    }                                  \
  } while (0)

#define SN_TRY(expr)                   \
  do {                                 \
    int _st = (expr);                  \
    if (_st != SN_OK) return _st;      \
  } while (0)

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Number of SMs of the current device (cached per process; single-GPU use).
int num_sms();

// Raises a kernel's dynamic shared-memory limit to `bytes` once per (device,
// kernel); later calls only look the pair up, so launches made while a stream
// is being captured issue no attribute calls.
int ensure_smem_limit(const void* fn, size_t bytes, const char* what);

inline unsigned int div_up(int64_t a, int64_t b) {
  return (unsigned int)((a + b - 1) / b);
}

// Grid size for a grid-stride kernel: enough blocks to cover n, capped at a
// whole number of waves over all SMs.
inline unsigned int stride_grid(int64_t n, int threads, int blocks_per_sm) {
  int64_t need = (n + threads - 1) / threads;
  int64_t cap = (int64_t)num_sms() * blocks_per_sm;
  if (need < 1) need = 1;
  return (unsigned int)(need < cap ? need : cap);
}

// ---------------------------------------------------------------------------
// device helpers
// ---------------------------------------------------------------------------
struct f3 {
  float x, y, z;
};

__device__ __forceinline__ f3 mk(float x, float y, float z) { return f3{x, y, z}; }

// Counter-based uniform random numbers in [0, 1): a 64-bit mix of
// (seed, stream, index).  Used only where the reference draws from
// torch.rand / torch.randint and the exact stream is not part of the
// contract (jitter, cell sampling).
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__device__ __forceinline__ float uniform01(uint64_t seed, uint64_t stream, uint64_t idx) {
  uint64_t h = mix64(seed ^ mix64(stream * 0x632BE59BD9B4E019ull + idx));
  return (float)(h >> 40) * (1.0f / 16777216.0f);  // 24 random bits
}
__device__ __forceinline__ uint32_t uniform_u32(uint64_t seed, uint64_t stream, uint64_t idx) {
  return (uint32_t)(mix64(seed ^ mix64(stream * 0x632BE59BD9B4E019ull + idx)) >> 32);
}

// torch.nn.Softplus(beta, threshold) forward and its derivative
// (torch/nn/modules/activation.py Softplus; ATen softplus kernel semantics).
__device__ __forceinline__ float softplus_fwd(float x, float beta, float threshold) {
  float bx = x * beta;
  return bx > threshold ? x : log1pf(expf(bx)) / beta;
}
__device__ __forceinline__ float softplus_grad(float x, float beta, float threshold) {
  float bx = x * beta;
  if (bx > threshold) return 1.0f;
  float z = expf(bx);
  return z / (z + 1.0f);
}
// Both at once (one exponential); the same values as the two functions above.
__device__ __forceinline__ void softplus_fwd_grad(float x, float beta, float threshold, float& y,
                                                  float& dy) {
  const float bx = x * beta;
  if (bx > threshold) {
    y = x;
    dy = 1.0f;
    return;
  }
  const float z = expf(bx);
  y = log1pf(z) / beta;
  dy = z / (z + 1.0f);
}
// 2^x and log2 x by the hardware approximations, subnormals as zero.
__device__ __forceinline__ float hw_exp2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float hw_log2(float x) {
  float r;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// Softplus through them, y = log(1 + z) / beta, z = exp(beta x): a subnormal z changes
// no bit of 1 + z, and the logarithm is taken of at least 1.  Against the accurate pair
// above the absolute error of y stays below 4e-9 for beta = 100 and z < 1, and
// within a few ulp beyond.  A select instead of a branch: past the threshold z may
// overflow, unread.
__device__ __forceinline__ float softplus_fast(float x, float beta, float inv_beta, float threshold) {
  constexpr float kLog2E = 1.4426950408889634f, kLn2 = 0.6931471805599453f;
  const float bx = x * beta;
  return bx > threshold ? x : hw_log2(1.0f + hw_exp2(bx * kLog2E)) * kLn2 * inv_beta;
}
__device__ __forceinline__ float hw_rcp(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// The same y and its derivative z / (1 + z), which is as small as z is: here z keeps
// its subnormals, and the reciprocal, of at least 1, is multiplied without a flush (the
// bits of __fdividef for every z from 0 to 2^31).
__device__ __forceinline__ void softplus_fwd_grad_fast(float x, float beta, float inv_beta,
                                                       float threshold, float& y, float& dy) {
  constexpr float kLn2 = 0.6931471805599453f;
  const float bx = x * beta;
  const float z = __expf(bx);
  const float u = 1.0f + z;
  const bool linear = bx > threshold;
  y = linear ? x : hw_log2(u) * kLn2 * inv_beta;
  dy = linear ? 1.0f : __fmul_rn(z, hw_rcp(u));
}
__device__ __forceinline__ float sigmoidf_(float x) { return 1.0f / (1.0f + expf(-x)); }

}  // namespace sn
