// Shared-memory barriers of the update kernels' stage rings: bulk copies
// complete on them, consumers wait on them for a bounded time.
#pragma once

#include <stdint.h>

namespace pfdtd {
namespace {

constexpr uint64_t kWaitLimitNs = 2000000000ull;  // 2 s per wait, far above any real wait

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Non-blocking test of the phase with the given parity.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}

// The waiting part of mbar_wait.  A bound under 1 ms (a watchdog set short)
// polls without blocking and reads the clock at every poll, since a blocking
// try_wait may itself sleep longer than such a bound; a longer bound blocks
// in try_wait and reads the clock every 256 polls.
__device__ __forceinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, uint64_t limit_ns) {
  const uint64_t t0 = global_ns();
  if (limit_ns < 1000000ull) {
    while (!mbar_test(bar, parity))
      if (global_ns() - t0 > limit_ns) return false;
    return true;
  }
  for (uint32_t i = 1;; ++i) {
    if (mbar_try(bar, parity)) return true;
    if ((i & 255) == 0 && global_ns() - t0 > limit_ns) return false;
  }
}

// Wait for the phase with the given parity, for at most limit_ns; false on
// expiry.  The common case in a streaming consumer, a phase already complete,
// costs one non-blocking test.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity,
                                          uint64_t limit_ns = kWaitLimitNs) {
  if (mbar_test(bar, parity)) return true;
  return mbar_wait_slow(bar, parity, limit_ns);
}

}  // namespace
}  // namespace pfdtd
