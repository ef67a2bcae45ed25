// cluster.cuh -- thread-block cluster primitives: the cluster barrier, the CTA's rank, and stores
// into the shared memory of the cluster's other CTAs (made visible by the barrier).
#pragma once

namespace dmrg {
namespace {

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ int cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return int(r);
}
__device__ __forceinline__ unsigned smem_addr(const void* p) {
  return unsigned(__cvta_generic_to_shared(p));
}
// the address in CTA `rank` of the cluster of the shared-memory address a of this CTA
__device__ __forceinline__ unsigned peer_addr(unsigned a, int rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void peer_store(unsigned addr, double a, double b) {
  asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" :: "r"(addr), "d"(a), "d"(b) : "memory");
}
__device__ __forceinline__ void peer_store(unsigned addr, double a) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" :: "r"(addr), "d"(a) : "memory");
}

}  // namespace
}  // namespace dmrg
