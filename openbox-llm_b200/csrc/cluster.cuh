// Thread-block clusters: the barrier of all threads of all CTAs, and reads of a peer CTA's shared memory.
#pragma once

#include <stdint.h>

namespace nsa {

// Every thread of every CTA of the cluster takes part.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t peer_addr(const void* p, int rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ int ld_peer_s32(const int* p, int rank) {
  int v;
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(peer_addr(p, rank)) : "memory");
  return v;
}
__device__ __forceinline__ float ld_peer_f32(const float* p, int rank) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(peer_addr(p, rank)) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_peer_f32x4(const float* p, int rank) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(peer_addr(p, rank)) : "memory");
  return v;
}

}  // namespace nsa
