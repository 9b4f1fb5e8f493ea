// tcgen05 (UMMA) and mbarrier helpers shared by the tensor-memory kernels.
#pragma once

#include "bbk_internal.cuh"

namespace bbk {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Shared-memory matrix descriptor, SWIZZLE_NONE K-major: start address,
// leading (k-direction, 128 B) and stride (row-direction) byte offsets,
// version 1.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t sbo) {
  constexpr uint64_t kLbo = 128 >> 4;
  return (static_cast<uint64_t>((saddr >> 4) & 0x3FFF)) | (kLbo << 16) |
         (static_cast<uint64_t>(sbo >> 4) << 32) | (1ull << 46);
}

__device__ __forceinline__ void umma_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
               : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t mbar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(done)
      : "r"(mbar), "r"(parity)
      : "memory");
  return done != 0;
}

// Bounded wait for phase `parity` of mbarrier `mbar`: false when it ran out
// (or another kernel of the factorization aborted).
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity, const DeviceState* st, unsigned long long timeout_ns) {
  unsigned long long t0 = 0;
  for (unsigned it = 1;; ++it) {
    if (mbar_try(mbar, parity)) return true;
    if ((it & 63u) == 0) {
      const unsigned long long now = globaltimer_ns();
      if (t0 == 0) t0 = now;
      if (now - t0 > timeout_ns || ld_relaxed_s32(&st->abort)) return false;
    }
  }
}

__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}

}  // namespace bbk
