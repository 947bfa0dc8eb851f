// Bulk copies global -> shared (cp.async.bulk) completing on an mbarrier.
#pragma once

namespace tcad {

__device__ __forceinline__ unsigned smem_addr(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}

// (one arrival: the expect_tx of the copies); make it visible to the async
// proxy with fence_async before the first copy
__device__ __forceinline__ void mbar_init(uint64_t* b, unsigned arrivals = 1) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(arrivals)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async;" ::: "memory"); }

__device__ __forceinline__ void mbar_expect(uint64_t* b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)),
               "r"(bytes)
               : "memory");
}

// n bytes, a multiple of 16, both addresses on 16-byte boundaries
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, unsigned n, uint64_t* b) {
  asm volatile(
      "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(n), "r"(smem_addr(b))
      : "memory");
}
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, unsigned n, uint64_t* b,
                                          uint64_t policy) {
  asm volatile(
      "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1], %2, [%3], %4;" ::"r"(smem_addr(dst)),
      "l"(src), "r"(n), "r"(smem_addr(b)), "l"(policy)
      : "memory");
}

__device__ __forceinline__ bool mbar_try(uint64_t* b, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_addr(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// wait for the phase, at most kBarrierNs of device time (a try suspends for a while);
// lost: no longer than a try.  A thread whose wait ran out does not wait for other
// copies, starts none, and waits once more for its own in flight before it returns.
__device__ __forceinline__ bool mbar_wait(uint64_t* b, unsigned parity, bool lost = false) {
  unsigned long long t0 = 0;
  for (unsigned i = 1; !mbar_try(b, parity); ++i) {
    if (lost) return false;
    if ((i & 15u) != 0u) continue;
    const unsigned long long now = globaltimer_ns();
    if (t0 == 0) t0 = now;
    if (now - t0 > kBarrierNs || i > (1u << 30)) return false;
  }
  return true;
}

}  // namespace tcad
