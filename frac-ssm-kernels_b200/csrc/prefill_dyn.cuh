#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace fracssm {

// out[rows, N] = x[rows, K] (rows x_sl elements apart) w[N, K]^T, all bf16.  A kernel launched behind it with programmatic
// stream serialisation may start at once and has to wait for it (griddepcontrol.wait) before it ends.
int prefill_dyn_launch(const void *x, int64_t x_sl, const void *w, void *out, int64_t rows, int64_t K, int64_t N,
                       cudaStream_t st);

}  // namespace fracssm
