// Submits whose kernels have to run one behind the other though they are on different batches: consecutive batches of one
// queue or of one GPU's share of a dispatcher call, which may carry packets of the same keypairs.
//
// Batches that stay in pinned memory have no copies that could overlap with each other's kernels, so they share one
// stream (batch_set_direct_stream) and are in order without more; a chain of events between streams costs 2.5 us a
// submit.  Batches that are copied run on streams of their own, and events order their kernels only.
#pragma once

#include <cuda_runtime.h>

#include "../../include/bnk_gpu.h"

#define BNK_INTERNAL __attribute__((visibility("hidden")))

// Where a batch's last submit ran, and how another one's kernels get behind its kernels.
struct SubmitOrder {
    cudaStream_t run; // bnk_wait waits for it, also after a submit that failed half way
    cudaEvent_t ev;   // behind the kernels, in front of the copies, if `recorded`
    bool recorded;

    // Before the submit queues anything.
    void begins(cudaStream_t s) {
        run = s;
        recorded = false;
    }
    // The last kernel is queued and copies follow.
    cudaError_t kernels_end() {
        const cudaError_t e = cudaEventRecord(ev, run);
        recorded = e == cudaSuccess;
        return e;
    }
    // This submit's kernels come next on its stream, behind those of p.  (Without an event in front of p's copies, because it
    // has none or because it failed before them: behind all that p has queued.)
    cudaError_t follow(const SubmitOrder &p) const {
        if (p.run == run) return cudaSuccess;
        const cudaError_t e = p.recorded ? cudaSuccess : cudaEventRecord(p.ev, p.run);
        return e != cudaSuccess ? e : cudaStreamWaitEvent(run, p.ev, 0);
    }
    // This submit failed, perhaps before it was behind p: who follows it shall be behind p all the same.
    static void failed_behind(const SubmitOrder &p) { (void)cudaStreamSynchronize(p.run); }
};

// Between the two calls, b's next submit starts its kernels behind those of `behind`'s last one (null: nothing in front).
BNK_INTERNAL int order_begin(bnk_batch *b, bnk_batch *behind);
BNK_INTERNAL void order_end(bnk_batch *b, int rc);
BNK_INTERNAL void batch_set_direct_stream(bnk_batch *b, cudaStream_t s); // outlives the batch's submits
BNK_INTERNAL cudaError_t order_stream_create(bnk_ctx *ctx, cudaStream_t *s);

template <typename F>
int submit_behind(bnk_batch *b, bnk_batch *behind, F submit) {
    int rc = order_begin(b, behind == b ? nullptr : behind); // its own earlier submit has been waited for
    if (rc == BNK_SUCCESS) rc = submit();
    order_end(b, rc);
    return rc;
}
