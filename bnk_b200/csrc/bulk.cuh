// Bulk copies between shared and global memory (a ring's on the device or the host's), by one thread; addresses and sizes are
// multiples of 16.  What comes in counts its bytes on an mbarrier of shared memory.  Over the link the copy engine of the SM
// asks for whole lines wherever the bytes start: 16,384 x 1440 B read 1456 bytes apart 488 us, in 16-byte pieces by the
// lanes of a warp 875 (1536 bytes apart 498 either way).
#pragma once

#include <stdint.h>

// How often a wait looks before it gives up.  A look that finds nothing takes 4 us, in which the warp sleeps, so that is half a
// second.  (A build for tests has it give up soon, and BNK_BULK_LOST set: copies of that many bytes are never asked for, which is
// what a link that has stopped looks like from here.)
#ifndef BNK_BULK_TURNS
#define BNK_BULK_TURNS (1u << 17)
#endif
__device__ __forceinline__ uint32_t shared_at(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint64_t *bar, uint32_t arrivals = 1) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(shared_at(bar)), "r"(arrivals) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(shared_at(bar)) : "memory");
}
__device__ __forceinline__ bool bar_test(uint64_t *bar, uint32_t parity) { // is the phase over?
    uint32_t over;
    asm volatile("{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(over)
                 : "r"(shared_at(bar)), "r"(parity)
                 : "memory");
    return over;
}
__device__ __forceinline__ void bar_expect(uint64_t *bar, uint32_t bytes) { // the phase ends when that many have come
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(shared_at(bar)), "r"(bytes) : "memory");
}
// False: it has not come after so many turns, which no link that works takes.
__device__ __forceinline__ bool bar_wait(uint64_t *bar, uint32_t parity) {
    for (uint32_t turn = 0; turn < BNK_BULK_TURNS; turn++) {
        uint32_t over;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                     : "=r"(over)
                     : "r"(shared_at(bar)), "r"(parity)
                     : "memory");
        if (over) return true;
    }
    return false;
}
__device__ __forceinline__ void bulk_in(void *smem, const void *gmem, uint32_t bytes, uint64_t *bar) {
#ifdef BNK_BULK_LOST
    if (bytes == BNK_BULK_LOST) return;
#endif
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(shared_at(smem)),
                 "l"(__cvta_generic_to_global(gmem)), "r"(bytes), "r"(shared_at(bar))
                 : "memory");
}
__device__ __forceinline__ void bulk_out(void *gmem, const void *smem, uint32_t bytes) { // counted per thread
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(__cvta_generic_to_global(gmem)), "r"(shared_at(smem)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_out_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_out_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); } // shared memory may change
__device__ __forceinline__ void bulk_out_read_but_last() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }
__device__ __forceinline__ void bulk_out_done() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }      // it is all where it belongs
__device__ __forceinline__ void bulk_fence() { asm volatile("fence.proxy.async;" ::: "memory"); }
// Between this thread's own accesses to shared memory and the bulk copies that follow.
__device__ __forceinline__ void bulk_fence_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
