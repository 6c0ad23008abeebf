// mbarriers of the warp-specialised tensor-core kernels (attention_tc.cu, gemm_pair.cu, skinny_gemm.cu, ssd_chunk.cu, router_tc.cu) and their bounded waits.
//
// A wait that runs out is an error of the kernel, never a slow neighbour: every role waits for the kernels in front of its own (griddepcontrol.wait)
// before it may block here.  The role then sets `stop`, which ends the other waits of the CTA, issues nothing more and runs to its end; the launch's
// word of wait_words() (pinned host memory) is set, and the host raises at its next launch or where it reads results (check_waits, kernel_status.cu).
#pragma once
#include <stdint.h>

namespace nxdi {

constexpr long long WAIT_LIMIT = 20000000000LL;     // SM clocks: about ten seconds

__device__ __forceinline__ uint32_t mbar_s32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar_s32(b)), "r"(n)); }
__device__ __forceinline__ void mbar_expect(uint64_t* b, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar_s32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar_s32(b)) : "memory"); }
// CLUSTER: arrivals may come from the other CTA of a pair
template <bool CLUSTER>
__device__ __forceinline__ bool mbar_try(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  if constexpr (CLUSTER)
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(mbar_s32(b)), "r"(parity) : "memory");
  else
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(mbar_s32(b)), "r"(parity) : "memory");
  return ok != 0u;
}
// false: gave up, or another role of the CTA did
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity, volatile int* stop, unsigned* word, long long limit = WAIT_LIMIT) {
  if (mbar_try<CLUSTER>(b, parity)) return true;
  const long long t0 = clock64();
  do {
    if (mbar_try<CLUSTER>(b, parity)) return true;
    if (*stop) return false;
  } while (clock64() - t0 < limit);
  *stop = 1;
  *reinterpret_cast<volatile unsigned*>(word) = 1u;
  __threadfence_system();
  return false;
}
// the same answer in all lanes of a warp that goes on with warp-wide instructions
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* b, uint32_t parity, volatile int* stop, unsigned* word) {
  return __all_sync(0xffffffffu, mbar_wait<CLUSTER>(b, parity, stop, word));
}

}  // namespace nxdi
