// team_sync.cuh -- mbarrier and bulk-copy helpers of the team kernels (inline PTX for sm_100a).
//
// Every wait is bounded: mbar_wait gives up after a number of polls and returns false.  The team kernels
// then wait (bounded again) for their copies in flight, set bit 0 of their error word and end the CTA, so a
// copy that never completes ends the launch with an error status that the host reads, not a hung GPU.
#pragma once
#include <cstdint>

namespace qcg {
namespace team {

// a wait for a bulk copy gives up after this many polls (each poll may suspend the thread for a while)
constexpr long long kWaitPolls = 1ll << 24;

__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ void mbar_init_fence()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// bulk copy of `bytes` (a multiple of 16; both addresses 16-byte aligned) from global to shared memory,
// completing a phase of `bar`
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}

// bounded wait for phase `parity` of `bar`; false when it gave up after `polls` polls
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, long long polls = kWaitPolls)
{
    for (long long n = 0; n < polls; ++n)
    {
        uint32_t done;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(smem_addr(bar)), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// After the wait for slot `slot` of the ring of three gave up: wait, bounded, for the copies still in flight -- that
// slot's and the ones after it, n in all -- so that none lands in this CTA's shared memory after it exited.
__device__ __forceinline__ void drain(uint64_t* full, int slot, uint32_t phase, int n)
{
    for (int x = 0; x < n; ++x)
    {
        mbar_wait(&full[slot], phase);
        if (++slot == 3)
        {
            slot = 0;
            phase ^= 1;
        }
    }
}

// one more warp is done with a slot (its reads come before, the slot's next copy after); the count before
__device__ __forceinline__ int count_done(int* done)
{
    int old;
    asm volatile("atom.acq_rel.cta.shared::cta.add.s32 %0, [%1], 1;" : "=r"(old) : "r"(smem_addr(done)) : "memory");
    return old;
}

// the barrier's memory may be reused for other data afterwards
__device__ __forceinline__ void mbar_inval(uint64_t* bar)
{
    asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// this thread's generic-proxy accesses to global and shared memory come before later bulk copies (async proxy)
__device__ __forceinline__ void fence_async()
{
    asm volatile("fence.proxy.async;" ::: "memory");
}

}   // namespace team

}   // namespace qcg
