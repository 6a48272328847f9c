#include "tmap.cuh"

#include <cuda_runtime.h>
#include <mutex>

#include "common.cuh"

namespace fracssm {

using EncodeFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                              const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                              CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                              CUtensorMapFloatOOBfill);

static EncodeFn encode_fn() {
  static EncodeFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeFn>(p);
  });
  return fn;
}

static int encode(CUtensorMap *map, const void *base, const cuuint64_t (&dims)[3], const cuuint64_t (&strides)[2],
                  uint32_t b0, uint32_t b1) {
  EncodeFn fn = encode_fn();
  if (!fn) return fail(FRACSSM_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || strides[0] % 16 != 0)
    return fail(FRACSSM_ERR_ARG, "TMA needs a 16-byte aligned base and row pitch");
  cuuint32_t box[3] = {b0, b1, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(base), dims, strides, box,
                  estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(FRACSSM_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", (int)r);
  return FRACSSM_OK;
}

int make_tmap_bf16_3d(CUtensorMap *map, const void *base, uint64_t d0, uint64_t d1, uint64_t d2,
                      uint32_t b0, uint32_t b1) {
  const cuuint64_t dims[3] = {d0, d1, d2}, strides[2] = {d0 * 2, d0 * d1 * 2};
  return encode(map, base, dims, strides, b0, b1);
}

int make_tmap_bf16_rows(CUtensorMap *map, const void *base, uint64_t d0, uint64_t d1, uint64_t pitch, uint32_t b0,
                        uint32_t b1) {
  const cuuint64_t dims[3] = {d0, d1, 1}, strides[2] = {pitch * 2, pitch * d1 * 2};
  return encode(map, base, dims, strides, b0, b1);
}

}  // namespace fracssm
