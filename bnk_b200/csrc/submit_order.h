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

// Between the two calls, b's next submit starts its kernels behind those of `behind`'s last one (null: nothing in front).
BNK_INTERNAL int order_begin(bnk_batch *b, bnk_batch *behind);
BNK_INTERNAL void order_end(bnk_batch *b);
BNK_INTERNAL void batch_set_direct_stream(bnk_batch *b, cudaStream_t s); // outlives the batch's submits
BNK_INTERNAL cudaError_t order_stream_create(bnk_ctx *ctx, cudaStream_t *s);

template <typename F>
int submit_behind(bnk_batch *b, bnk_batch *behind, F submit) {
    int rc = order_begin(b, behind == b ? nullptr : behind); // its own earlier submit has been waited for
    if (rc == BNK_SUCCESS) rc = submit();
    order_end(b);
    return rc;
}
