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

// Waits for phase `parity` of `mbar`, aborted or not, until a second after t0.
// The copying and the MMA-issuing role of a tensor-memory kernel end with it,
// whether they came to their end or gave up: what they issued is done before
// the CTA gives up shared and tensor memory, also when only another role gave
// up, and however short the caller's own wait limit is.
__device__ __forceinline__ void mbar_finish(uint32_t mbar, uint32_t parity, unsigned long long t0) {
  while (!mbar_try(mbar, parity) && globaltimer_ns() - t0 < 1000000000ull) {
  }
}

__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}

// One lane of the (converged) warp.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(p));
  return p != 0;
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const unsigned char* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// 16 rows x 8 columns of an accumulator: v[0], v[1] row lane / 4, v[2], v[3]
// row lane / 4 + 8, at columns 2 (lane % 4) and the next.
__device__ __forceinline__ void tmem_ld16x8(uint32_t addr, int (&v)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "r"(addr));
}

// 32 rows (one per lane) x 32 columns of an accumulator.
__device__ __forceinline__ void tmem_ld32x32(uint32_t addr, int (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
        "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(addr));
}

// Tile t of an upper triangle of tm x tm tiles (row I, column J >= I): in
// strips of kStrip tile columns, row by row within a strip, so the CTAs that
// run together share a few row and column blocks of operands in L2.
constexpr int kStrip = 12;  // 12 x 12 tiles for 148 CTAs
__device__ __forceinline__ void strip_tile(int t, int tm, int& I, int& J) {
  constexpr int kTri = kStrip * (kStrip + 1) / 2;
  auto before = [](int q) { return kStrip * kStrip * (q * (q - 1) / 2) + kTri * q; };  // tiles of the strips < q
  int q = static_cast<int>(sqrt(2.0 * t) / kStrip);
  while (q > 0 && before(q) > t) --q;
  while (before(q + 1) <= t) ++q;
  const int j0 = q * kStrip, w = min(kStrip, tm - j0);
  int u = t - before(q);
  if (u < w * j0) {
    I = u / w;
    J = j0 + u % w;
    return;
  }
  u -= w * j0;
  int j = 0;
  while ((j + 1) * (j + 2) / 2 <= u) ++j;
  I = j0 + u - j * (j + 1) / 2;
  J = j0 + j;
}

}  // namespace bbk
