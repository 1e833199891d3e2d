// Blocks of a thread-block cluster and their shared memory.
#pragma once

#include "common.cuh"

namespace sn {

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// The cluster's barrier in its two halves; every thread of the cluster takes part
// in each.  A block's shared memory may be stored to only once that block runs:
// kernels arrive when they start and wait before their first remote store, and
// arrive and wait once more between the stores and their use.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// v to address `at` (this block's shared memory) of block `rank` of the cluster.
__device__ __forceinline__ void st_cluster(double* at, uint32_t rank, double v) {
  uint32_t local = (uint32_t)__cvta_generic_to_shared(at), remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(remote), "d"(v) : "memory");
}

}  // namespace sn
