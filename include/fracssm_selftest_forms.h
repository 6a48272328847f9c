/*
 * fracssm_selftest_forms.h -- further test-only entry points of libfracssm_selftest.so (see fracssm_selftest.h): a product
 * call in a form that its own rule would not take here.  None has a counterpart in quorbix/frac-ssm-kernels.
 */
#ifndef FRACSSM_SELFTEST_FORMS_H
#define FRACSSM_SELFTEST_FORMS_H

#include "fracssm.h"

#ifdef __cplusplus
extern "C" {
#endif

/*
 * fracssm_decode_layers as a kernel per stage (one_kernel 0) or as one kernel (up to 32 sequences) of `blocks` blocks, 0: one
 * per SM.  The results are the same bits in every form and with every number of blocks.
 */
int fracssm_selftest_decode_layers(const uint64_t *layer_ptrs, const float *layer_nums, int64_t layers, const void *hidden_in,
                                   void *hidden_out, void *workspace, size_t workspace_bytes, int64_t B, int64_t hidden,
                                   int64_t H, int64_t R, int64_t M, int64_t K, void *stream, int one_kernel, int blocks);
/*
 * The one-kernel form whose block 0 waits at the `barrier`-th meeting of the blocks (4 a layer, less one) for the arrivals
 * of the next one, which needs its own.  After wait_ns nanoseconds it gives up, the kernel returns by itself, fracssm_decode_layers_status reports
 * FRACSSM_ERR_WAIT and all outputs are NaN, also where the other blocks have finished.
 */
int fracssm_selftest_decode_wait_limit(const uint64_t *layer_ptrs, const float *layer_nums, int64_t layers,
                                       const void *hidden_in, void *hidden_out, void *workspace, size_t workspace_bytes,
                                       int64_t B, int64_t hidden, int64_t H, int64_t R, int64_t M, int64_t K, void *stream,
                                       int barrier, unsigned long long wait_ns);
/*
 * The projection of fracssm_prefill_conv_dyn alone, dyn [rows, cols] = x [rows, K] w [cols, K]^T, where one load of every 128
 * rows is left out (not the wait for it).  After wait_ns nanoseconds the kernel carries on and returns, and dyn is NaN.
 */
int fracssm_selftest_prefill_dyn_wait_limit(const void *x, int64_t x_sl, const void *w, void *dyn, int64_t rows, int64_t K,
                                            int64_t cols, unsigned long long wait_ns, void *stream);

#ifdef __cplusplus
}
#endif
#endif /* FRACSSM_SELFTEST_FORMS_H */
