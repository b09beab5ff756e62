// Thread-block clusters: rank, size, the hardware barrier and addresses in the shared memory
// of another CTA of the cluster.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace umapb {
namespace cluster {

__device__ __forceinline__ uint32_t rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

__device__ __forceinline__ uint32_t size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}

// All threads of all CTAs; what a thread wrote before is visible to every thread after.
// Called with the warp converged.
__device__ __forceinline__ void barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ uint32_t smem_address(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// shared::cluster address of the object at the same offset in CTA `rank`
__device__ __forceinline__ uint32_t peer(uint32_t smem, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem), "r"(rank));
  return r;
}

}  // namespace cluster
}  // namespace umapb
