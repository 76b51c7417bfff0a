// pm_bulk.cuh — bulk (TMA) copies from global to shared memory under
// mbarriers, with bounded waits.
#ifndef PM_BULK_CUH
#define PM_BULK_CUH

#include <cuda_runtime.h>

#include <cstdint>

namespace pm {

// non-blocking polls of a wait before it gives up (a few hundred ms)
constexpr int kMaxPolls = 1 << 22;

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count)
               : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// one thread: arm the barrier for the bytes of the copies that follow
__device__ __forceinline__ void bulk_expect(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
}
// one thread: start a copy global -> shared (16-byte boundaries and sizes)
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, uint32_t bytes,
                                          uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

// arm the barrier and start one copy
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes,
                                          uint64_t *bar) {
  bulk_expect(bar, bytes);
  bulk_copy(dst, src, bytes, bar);
}

__device__ __forceinline__ bool mbar_test_wait(uint64_t *bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return done != 0;
}

// Bounded wait by the whole warp (at most `polls` non-blocking tests); true
// when the phase completed.  The result is warp-uniform (every lane has
// observed the completion itself, so every lane's later shared-memory reads
// are ordered after the copy).
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, int polls) {
  for (int it = 0; it < polls; ++it)
    if (__all_sync(0xffffffffu, mbar_test_wait(bar, parity))) return true;
  return false;
}

}  // namespace pm

#endif
