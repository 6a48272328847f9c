// Test-only entry points (built into libfracssm_selftest.so, not into the product library): a decode step in either of its
// forms, the one-kernel form with any number of blocks or with a wait that runs out; the prefill's projection with one that does.
#include "common.cuh"
#include "fracssm_selftest_forms.h"
#include "prefill_dyn.cuh"

extern "C" int fracssm_selftest_decode_layers(const uint64_t *layer_ptrs, const float *layer_nums, int64_t layers,
                                              const void *hidden_in, void *hidden_out, void *workspace,
                                              size_t workspace_bytes, int64_t B, int64_t hidden, int64_t H, int64_t R,
                                              int64_t M, int64_t K, void *stream, int one_kernel, int blocks) {
  using namespace fracssm;
  if (one_kernel && (B > 32 || blocks < 0 || blocks > 1024))
    return fail(FRACSSM_ERR_ARG, "selftest_decode_layers: one kernel is for up to 32 sequences");
  DecodeForm how;
  how.form = one_kernel ? DecodeForm::kOneKernel : DecodeForm::kStages;
  how.blocks = blocks;
  return decode_layers_launch(layer_ptrs, layer_nums, layers, hidden_in, hidden_out, workspace, workspace_bytes, B, hidden, H,
                              R, M, K, stream, how);
}

extern "C" int fracssm_selftest_decode_wait_limit(const uint64_t *layer_ptrs, const float *layer_nums, int64_t layers,
                                                  const void *hidden_in, void *hidden_out, void *workspace,
                                                  size_t workspace_bytes, int64_t B, int64_t hidden, int64_t H, int64_t R,
                                                  int64_t M, int64_t K, void *stream, int barrier,
                                                  unsigned long long wait_ns) {
  using namespace fracssm;
  if (B > 32 || barrier < 1 || wait_ns > tile_default_wait_ns())
    return fail(FRACSSM_ERR_ARG, "selftest_decode_wait_limit: up to 32 sequences, a barrier and a limit");
  DecodeForm how;
  how.form = DecodeForm::kOneKernel;
  how.wait_ns = wait_ns;
  how.lost = barrier;
  return decode_layers_launch(layer_ptrs, layer_nums, layers, hidden_in, hidden_out, workspace, workspace_bytes, B, hidden, H,
                              R, M, K, stream, how);
}

extern "C" int fracssm_selftest_prefill_dyn_wait_limit(const void *x, int64_t x_sl, const void *w, void *dyn, int64_t rows,
                                                       int64_t K, int64_t cols, unsigned long long wait_ns, void *stream) {
  using namespace fracssm;
  if (wait_ns > tile_default_wait_ns()) return fail(FRACSSM_ERR_ARG, "selftest_prefill_dyn_wait_limit: the limit");
  return prefill_dyn_launch(x, x_sl, w, dyn, rows, K, cols, (cudaStream_t)stream, wait_ns, true);
}
