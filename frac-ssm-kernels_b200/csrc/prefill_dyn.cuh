#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace fracssm {

// out[rows, N] = x[rows, K] (rows x_sl elements apart) w[N, K]^T, all bf16.  A kernel launched behind it with programmatic
// stream serialisation may start at once and has to wait for it (griddepcontrol.wait) before it ends.  Rows whose sums had to
// wait for longer than wait_ns are NaN; `withhold` (self-test) makes that happen, by a load that is left out.
int prefill_dyn_launch(const void *x, int64_t x_sl, const void *w, void *out, int64_t rows, int64_t K, int64_t N,
                       cudaStream_t st, uint64_t wait_ns = tile_default_wait_ns(), bool withhold = false);

}  // namespace fracssm
