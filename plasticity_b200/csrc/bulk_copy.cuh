// bulk_copy.cuh -- cp.async.bulk (global to shared memory) and the barriers it reports to.
#pragma once
#include <cstdint>

namespace pfem {

constexpr long long kBulkWaitLimit = 1ll << 20;  // polls of a barrier before a kernel gives up

__device__ __forceinline__ uint32_t bulk_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bulk_bar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
// After the inits, before the first copy.
__device__ __forceinline__ void bulk_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// This thread's accesses of shared memory before the copies that follow.
__device__ __forceinline__ void bulk_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ bool bulk_bar_poll(uint32_t bar, uint32_t phase, long long polls) {
  for (long long it = 0; it < polls; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar), "r"(phase)
        : "memory");
    if (done) return true;
  }
  return false;
}
// False, with *err set, when the phase has not completed within the limit.  Its copies may
// still be on their way then, into shared memory that is another CTA's once this one has
// left, so they get the limit once more before the caller is told.
__device__ __forceinline__ bool bulk_bar_wait(uint32_t bar, uint32_t phase, int* err, long long polls = kBulkWaitLimit,
                                              long long drain = kBulkWaitLimit) {
  if (bulk_bar_poll(bar, phase, polls)) return true;
  atomicExch(err, 1);
  bulk_bar_poll(bar, phase, drain);
  return false;
}
__device__ __forceinline__ void bulk_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Both addresses and the size are multiples of 16 bytes.
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// The same, with the lines marked for early eviction: what is streamed once should not
// push what is gathered out of L2.
__device__ __forceinline__ void bulk_copy_first(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .b64 pol;\n\tcreatepolicy.fractional.L2::evict_first.b64 pol, 1.0;\n\t"
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], pol;\n\t}\n" ::
          "r"(dst), "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}

}  // namespace pfem
