// Thread-block clusters in plain PTX: this CTA's rank, a barrier of all CTAs, and accesses to another CTA's shared memory by
// 32-bit addresses.  Such an access lies behind a barrier of the whole cluster, without which that CTA need not have started, and in
// front of one, without which it may have left.
#pragma once
#include <stdint.h>

namespace ds41 {

__device__ __forceinline__ uint32_t shared_addr(const void *p) { return uint32_t(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// All threads of all CTAs: what each has done before is seen by the others behind it.
__device__ __forceinline__ void cluster_barrier() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The address of CTA `rank`'s copy of a shared variable.
__device__ __forceinline__ uint32_t peer_addr(const void *p, int rank) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(shared_addr(p)), "r"(rank));
  return a;
}
__device__ __forceinline__ uint32_t peer_load_u32(uint32_t at) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
  return v;
}
__device__ __forceinline__ uint4 peer_load_u128(uint32_t at) {
  uint4 v;
  asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
  return v;
}
__device__ __forceinline__ void peer_store_u64(uint32_t at, unsigned long long v) {
  asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(at), "l"(v) : "memory");
}

}  // namespace ds41
