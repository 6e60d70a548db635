// TMA tensor maps of the fp16 and fp32 operand arrays (host side).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace ac {

// 3-D map over a row-major [batch, rows, cols] array of fp16 (elem 2) or fp32 (elem 4): boxes of 128 bytes of columns (the
// 128-byte swizzle) x box_rows rows; what lies past `rows` and `cols` is zero-filled.
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);
inline bool make_map128(CUtensorMap* map, const void* base, int elem, int64_t cols, int64_t rows, int64_t batch, int64_t ld,
                        int64_t batch_stride, int box_rows) {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  if (!fn) return false;
  cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)batch};
  cuuint64_t strides[2] = {(cuuint64_t)(ld * elem), (cuuint64_t)(batch_stride * elem)};
  cuuint32_t box[3] = {(cuuint32_t)(128 / elem), (cuuint32_t)box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return fn(map, elem == 2 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
inline bool make_map16(CUtensorMap* map, const void* base, int64_t cols, int64_t rows, int64_t batch, int64_t ld, int64_t batch_stride,
                       int box_rows) {
  return make_map128(map, base, 2, cols, rows, batch, ld, batch_stride, box_rows);
}

}  // namespace ac
