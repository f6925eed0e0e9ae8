// k_bulk.cuh -- bulk asynchronous copies global -> shared with an mbarrier (sm_90+ PTX).
#pragma once
#include <cuda_runtime.h>

namespace fcb {

__device__ __forceinline__ unsigned smem_u32(const void* p)
{
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
// One thread: expect `bytes` on the barrier (of all copies of the phase) ...
__device__ __forceinline__ void bulk_expect(unsigned long long* bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
// ... and start a copy (addresses and size multiples of 16 bytes) that completes on it.
__device__ __forceinline__ void bulk_copy(unsigned long long* bar, void* dst, const void* src, unsigned bytes)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
// Wait for phase `parity` of the barrier to complete, at most `limit` polls.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity, int limit)
{
    for (int i = 0; i < limit; i++) {
        unsigned done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
// Polls of a staging wait before the CTA gives up (each poll may suspend the thread
// for a while in hardware): far beyond any copy of a few KB, short of a hang.
constexpr int BULK_WAIT_LIMIT = 1 << 20;

// Whether this thread saw the CTA's staging copies (phase 0 of the barrier) arrive.  A translation
// unit that defines FCB_STAGE_LOST waits all the same but takes them for lost (tests of that path).
__device__ __forceinline__ bool stage_arrived(unsigned long long* bar)
{
    const bool arrived = mbar_wait(bar, 0u, BULK_WAIT_LIMIT);
#ifdef FCB_STAGE_LOST
    return false;
#else
    return arrived;
#endif
}

}  // namespace fcb
