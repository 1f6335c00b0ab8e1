// Shared-memory barriers (mbarrier) with bounded waits, used by the kernels whose warps have roles.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace dlspm {

constexpr unsigned kWaitLimit = 1u << 20;  // polls of an mbarrier (a quarter of a microsecond apart) before the kernel gives up

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: false after kWaitLimit polls (the caller records the failure and leaves).
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, unsigned parity)
{
    for (unsigned i = 0; i < kWaitLimit; i++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void mbar_arrive(unsigned long long *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Bounded wait that also gives up when another thread of the block has raised `abort`.
__device__ __forceinline__ bool mbar_wait_or_abort(unsigned long long *bar, unsigned parity, volatile int *abort)
{
    for (unsigned i = 0; i < kWaitLimit; i++) {
        if (mbar_try_wait(bar, parity)) return true;
        // a waiting warp must not take issue slots from the warps that compute
        if (i >= 4u) __nanosleep(i < 64u ? 64u : 256u);
        if ((i & 63u) == 63u && *abort) return false;
    }
    return false;
}

}  // namespace dlspm
