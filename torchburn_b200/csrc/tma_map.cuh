// Descriptions of row-major matrices for the TMA engine, and its two-dimensional copy into shared memory.
#pragma once

#include <climits>

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace tb {

#ifdef __CUDACC__
// The box from column x, row y on; x on a 16-byte boundary.  Columns and rows outside the matrix are zeros.
__device__ __forceinline__ void tma_box(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x),
               "r"(y), "r"(bar)
               : "memory");
}
#endif

using TmaEncode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
// The driver's call, or null when it lacks it.
inline TmaEncode tma_encoder() {
  static const TmaEncode encode = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &found) != cudaSuccess || found != cudaDriverEntryPointSuccess) fn = nullptr;
    return reinterpret_cast<TmaEncode>(fn);
  }();
  return encode;
}

// False when the matrix cannot be described (alignment, sizes) or the driver lacks the call.
inline bool tma_matrix_map(CUtensorMap* map, CUtensorMapDataType type, const void* base, int64_t cols, int64_t rows, int64_t stride_bytes, int box_cols,
                           int box_rows, CUtensorMapSwizzle swizzle) {
  const TmaEncode encode = tma_encoder();
  if (!encode || rows < 1 || rows > INT_MAX) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)stride_bytes};
  const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows}, steps[2] = {1, 1};
  return encode(map, type, 2, const_cast<void*>(base), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace tb
