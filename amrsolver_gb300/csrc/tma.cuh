// mbarrier helpers in inline PTX for sm_103a with a bounded wait: after
// MBAR_SPIN_LIMIT polls it gives up and reports failure to the caller, which
// raises an error flag the host reads, instead of hanging the GPU.
#pragma once
#include <cstdint>

namespace amrs {

constexpr long long MBAR_SPIN_LIMIT = 1ll << 26;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Returns false if the phase did not complete within `limit` polls.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity,
                                          long long limit = MBAR_SPIN_LIMIT) {
  const uint32_t a = smem_u32(bar);
  for (long long it = 0; it < limit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

}  // namespace amrs
