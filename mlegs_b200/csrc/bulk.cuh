// mbarrier and bulk-copy (cp.async.bulk) helpers of the pipelined kernels.  Every
// wait is bounded: a kernel whose wait runs out raises an error word, waits
// (bounded again) for the copies it issued and returns.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace mlegs {
namespace bulk {

constexpr uint64_t WAIT_CYCLES = 2000000000ull;  // about one second of SM cycles

__device__ __forceinline__ uint32_t sa_of(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(sa_of(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sa_of(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(sa_of(bar)) : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(sa_of(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Waits for the phase of `parity`; false after WAIT_CYCLES.
__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t parity) {
    if (bar_try(bar, parity)) return true;
    const uint64_t t0 = (uint64_t)clock64();
    while (!bar_try(bar, parity))
        if ((uint64_t)clock64() - t0 > WAIT_CYCLES) return false;
    return true;
}
__device__ __forceinline__ bool bar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(sa_of(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// The same with the caller's limit (0: WAIT_CYCLES), which is polled: try_wait may suspend
// the thread for longer than a limit of a few cycles.  The clock is read before the
// barrier, so a limit of one cycle runs out in every wait.
__device__ __forceinline__ bool bar_wait(uint64_t* bar, uint32_t parity, uint64_t limit) {
    if (limit == 0) return bar_wait(bar, parity);
    const uint64_t t0 = (uint64_t)clock64();
    do {
        if ((uint64_t)clock64() - t0 > limit) return false;
    } while (!bar_test(bar, parity));
    return true;
}
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(sa_of(dst)),
        "l"(src), "r"(bytes), "r"(sa_of(bar))
        : "memory");
}

// 16-byte copies of the calling thread, and its arrival once those so far have landed.
__device__ __forceinline__ void copy16_async(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa_of(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy16_arrive(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(sa_of(bar)) : "memory");
}

}  // namespace bulk
}  // namespace mlegs
