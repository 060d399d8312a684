/*
 * mc_pdlp_testing.h -- test hooks of the PDLP engine (no counterpart in the
 * reference; not part of the solver API).
 *
 * They let the host-side failure paths be exercised without faulting a GPU.
 */
#ifndef MC_PDLP_TESTING_H
#define MC_PDLP_TESTING_H

#include "mc_pdlp.h"

#ifdef __cplusplus
extern "C" {
#endif

/* The next `count` allocations of a context's device arena or of a network's
 * workspace fail as if cudaMalloc had returned cudaErrorMemoryAllocation: the
 * call returns MC_ERR_OUT_OF_MEMORY and no device memory is touched.  0 disarms. */
int mc_test_inject_alloc_failures(int count);

/* How many polls the waits inside the context's cooperative kernels take before
 * a kernel gives up and its call returns MC_ERR_CUDA: at a barrier of the grid,
 * and for one entry that another block writes.  0 restores a default (seconds).
 * A few polls make an ordinary wait run out.  The Ruiz passes' barrier adds
 * polls_per_nonzero (default 2) for every nonzero of the matrix. */
int mc_test_set_wait_limits(mc_pdlp_ctx* ctx, unsigned barrier_polls, unsigned entry_polls,
                            unsigned polls_per_nonzero);

/* In the persistent loop's form of one block per SM this block behaves as if a
 * wait of its had run out before its first gather: it waits for nothing and
 * goes on with whatever it reads, until the next reduction.  -1: none. */
int mc_test_fail_block(mc_pdlp_ctx* ctx, int block);

#ifdef __cplusplus
}
#endif

#endif
