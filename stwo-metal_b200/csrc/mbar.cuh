// Shared-memory addresses and bounded mbarrier waits (sm_100a).
//
// Every wait polls at most a given number of times (kStreamSpin by default);
// one that runs out returns false, and its kernel sets an error word, waits
// (bounded) for its own work in flight and leaves.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/stwo_b200.h"

namespace stwo_b200 {

constexpr uint32_t kStreamSpin = STWO_B200_STREAM_SPIN_DEFAULT;  // try_wait polls before giving up

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
// Waits for phase `parity` of `bar`; false when `limit` polls ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t limit = kStreamSpin) {
  const uint32_t a = smem_addr(bar);
  for (uint32_t it = 0; it < limit; it++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

}  // namespace stwo_b200
