// Submits whose kernels have to run one behind the other though they are on different batches: consecutive batches of one
// queue or of one GPU's share of a dispatcher call, which may carry packets of the same keypairs.  Copies on either side
// of the kernels stay free to overlap.
#pragma once

#include "../../include/bnk_gpu.h"

// Between the two calls, b's next submit starts its kernels behind those of `behind`'s last one (null: nothing to wait
// for) and leaves a mark of its own.  A batch keeps its mark until its next submit between the two.
__attribute__((visibility("hidden"))) int order_begin(bnk_batch *b, bnk_batch *behind);
__attribute__((visibility("hidden"))) void order_end(bnk_batch *b);

template <typename F>
int submit_behind(bnk_batch *b, bnk_batch *behind, F submit) {
    int rc = order_begin(b, behind == b ? nullptr : behind); // its own earlier submit is in front on the same stream
    if (rc == BNK_SUCCESS) rc = submit();
    order_end(b);
    return rc;
}
