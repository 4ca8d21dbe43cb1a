// tcgen05, mbarrier and bulk-copy primitives shared by the tensor-core correlation kernels
// (iq_corr_tc.cu, iq_corr_tz.cu). Every wait is bounded in time.
#pragma once

#include <cuda_fp16.h>

#include "iq_internal.h"

namespace {

constexpr unsigned long long TC_WAIT_NS = 2000000000ull; // bound of every wait

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Shared-memory matrix descriptor, no swizzle: start, leading (K) and stride (M/N) byte
// offsets in 16-byte units, descriptor version 1 at bit 46.
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}

// Wait for the phase of parity `parity` to complete; false after TC_WAIT_NS.
__device__ bool mbar_wait(uint32_t bar, uint32_t parity) {
  if (mbar_test(bar, parity)) return true;
  const unsigned long long t0 = globaltimer();
  for (uint32_t it = 1;; ++it) {
    if (mbar_test(bar, parity)) return true;
    if ((it & 63u) == 0 && globaltimer() - t0 > TC_WAIT_NS) return false;
  }
}

// mbar_wait that adds the cycles it spent to *acc when profiling
__device__ __forceinline__ bool mbar_wait_t(uint32_t bar, uint32_t parity, bool prof,
                                            long long& acc) {
  if (!prof) return mbar_wait(bar, parity);
  const long long t = clock64();
  const bool ok = mbar_wait(bar, parity);
  acc += clock64() - t;
  return ok;
}

__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes,
                                         uint32_t bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(dst),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   bar)
               : "memory");
}

// v * scale = hi + lo, both FP16 (round to nearest even)
__device__ __forceinline__ void f16_split(float v, float scale, uint16_t& hi, uint16_t& lo) {
  const float x = v * scale;  // a power of two: exact
  const __half h = __float2half_rn(x);
  const __half l = __float2half_rn(__fsub_rn(x, __half2float(h)));
  hi = __half_as_ushort(h);
  lo = __half_as_ushort(l);
}

__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                        uint32_t acc) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ bool in_box(const TcBox& b, int64_t x, int64_t y, int64_t z) {
  return x >= b.lo[0] && x < b.hi[0] && y >= b.lo[1] && y < b.hi[1] && z >= b.lo[2] &&
         z < b.hi[2];
}

}  // namespace
