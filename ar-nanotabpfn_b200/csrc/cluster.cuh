// Shared memory of the CTAs of a thread-block cluster: addresses, counted stores, mbarrier polls.
#pragma once
#include "common.cuh"

namespace artab {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t map_to_rank(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ bool mbar_try(uint32_t b, uint32_t parity) {  // may suspend the thread for a while
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(b), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool mbar_test(uint32_t b, uint32_t parity) {  // never suspends
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(b), "r"(parity)
      : "memory");
  return ok != 0;
}
// `n` consecutive floats into a shared-memory array of one CTA of the cluster, counted by its barrier
template <int N>
__device__ __forceinline__ void st_async(uint32_t addr, const float* v, uint32_t bar) {
  if constexpr (N == 1)
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(addr), "f"(v[0]),
                 "r"(bar)
                 : "memory");
  else if constexpr (N == 2)
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(addr),
                 "f"(v[0]), "f"(v[1]), "r"(bar)
                 : "memory");
  else
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
                 "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "r"(bar)
                 : "memory");
}

}  // namespace artab
