// Panels of 64 bf16 columns of a row-major matrix by TMA, with the tensor core's 128-byte swizzle on the way.
#pragma once

#include "dense.cuh"
#include "tma_map.cuh"

namespace tb {

#ifdef __CUDACC__
// The panel from column x, row y on; x on a 16-byte boundary.  Columns and rows outside the matrix are zeros.
__device__ __forceinline__ void tma_panel(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) { tma_box(dst, map, x, y, bar); }
#endif

// Panels of `panel_rows` rows; false when the matrix cannot be described (alignment, sizes) or the driver lacks the call.
inline bool tma_panel_map(CUtensorMap* map, const void* base, int64_t cols, int64_t rows, int64_t stride, int panel_rows) {
  return tma_matrix_map(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base, cols, rows, stride * 2, 64, panel_rows, CU_TENSOR_MAP_SWIZZLE_128B);
}

}  // namespace tb
