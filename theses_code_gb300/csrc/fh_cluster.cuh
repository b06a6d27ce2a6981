// fh_cluster.cuh -- one-sided messages between the CTAs of a cluster: a store
// into another CTA's shared memory that counts its bytes on an mbarrier there
// (st.async).  The receiver arms the barrier with the bytes of a phase, waits
// (bounded, fh_mbar_wait) and reads its own shared memory; no cluster barrier
// and no fence, which would also wait for the sender's stores to global memory.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "fh_sm100.cuh"

// Address of this CTA's shared-memory address in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t fh_mapa(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// Stores 8 bytes at a cluster address and completes them on the mbarrier there.
__device__ __forceinline__ void fh_st_async8(uint32_t addr, unsigned long long bits, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr), "l"(bits),
               "r"(bar)
               : "memory");
}
__device__ __forceinline__ void fh_st_async8(uint32_t addr, float2 v, uint32_t bar) {
  fh_st_async8(addr, ((unsigned long long)__float_as_uint(v.y) << 32) | __float_as_uint(v.x), bar);
}
__device__ __forceinline__ void fh_st_async8(uint32_t addr, double v, uint32_t bar) {
  fh_st_async8(addr, (unsigned long long)__double_as_longlong(v), bar);
}
