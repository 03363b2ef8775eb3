// Tensor maps for bulk tensor copies: the driver's encoder, and the map of a paged key or value cache.
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace ms {

using TensorMapEncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                       const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                       CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline int tensor_map_encoder(TensorMapEncodeFn* out) {
  static TensorMapEncodeFn fn = nullptr;
  if (fn == nullptr) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    MS_CHECK_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres));
    MS_CHECK_ARG(ptr != nullptr && qres == cudaDriverEntryPointSuccess, "the driver has no cuTensorMapEncodeTiled");
    fn = reinterpret_cast<TensorMapEncodeFn>(ptr);
  }
  *out = fn;
  return 0;
}

// A bfloat16 cache [pages, kv heads, page_size, d] (d = 64 or 128) as [groups of 8 rows][d / 64 parts of a row][8 rows][64]: one
// copy brings `box_rows` rows (a multiple of 8) of one page and head, each part of a group a block swizzled in 128 bytes. Coordinates: 0, 0, 0 and the
// group of rows that the copy begins with; groups past the pool's end read as zeros.
inline int cache_tensor_map(CUtensorMap* map, const void* pool, long long rows, int d, int box_rows) {
  TensorMapEncodeFn encode;
  if (int rc = tensor_map_encoder(&encode)) return rc;
  const cuuint64_t dims[4] = {64, 8, (cuuint64_t)(d / 64), (cuuint64_t)(rows / 8)};
  const cuuint64_t strides[3] = {(cuuint64_t)d * 2, 128, (cuuint64_t)d * 2 * 8};
  const cuuint32_t box[4] = {64, 8, (cuuint32_t)(d / 64), (cuuint32_t)(box_rows / 8)};
  const cuuint32_t elem[4] = {1, 1, 1, 1};
  const CUresult res = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(pool), dims, strides, box, elem,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  MS_CHECK_ARG(res == CUDA_SUCCESS, "encoding a cache's tensor map failed with code %d (%lld rows of %d)", (int)res, rows, d);
  return 0;
}

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %3, %3, %4}], [%2];\n"
      ::"r"(dst), "l"(map), "r"(bar), "r"(0), "r"(c3) : "memory");
}

}  // namespace ms
