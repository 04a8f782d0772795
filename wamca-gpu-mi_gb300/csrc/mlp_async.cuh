// mlp_async.cuh -- bulk asynchronous copies (TMA) into shared memory and the
// mbarrier they complete on.
#pragma once

#include <cstdint>

namespace mlp {

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// One mbarrier phase with `count` arrivals; visible to the async proxy after
// the fence (and to the other threads after a CTA barrier).
__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// Orders this thread's ordinary shared-memory accesses before later bulk
// copies to the same bytes.
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Copies `bytes` (a multiple of 16) from global to shared memory, both 16-byte
// aligned; completion is counted on `bar`.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}

// Waits for phase `parity` of the barrier, at most `tries` polls suspended for
// a microsecond or so each (kMbarTries: far longer than any copy takes); false
// if it did not complete.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int tries) {
  const uint32_t a = smem_addr(bar);
  for (int q = 0; q < tries; q++) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 1000;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

}  // namespace mlp
