// Tensor maps of row-major arrays of four-byte values, and the TMA copies of their boxes.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include "common.h"

namespace rxmet {

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link against the driver library); null where there is none.
using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                 const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline EncodeTiled encodeTiled() {
    static EncodeTiled fn = [] {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult status = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &status) != cudaSuccess ||
            status != cudaDriverEntryPointSuccess)
            ptr = nullptr;
        return reinterpret_cast<EncodeTiled>(ptr);
    }();
    return fn;
}

constexpr int kBoxRows = 32, kBoxCols = 32;
constexpr uint32_t kBoxBytes = kBoxRows * kBoxCols * 4;

// [rows][cols], 16-byte aligned, cols a multiple of 4; what lies beyond the array reads as zero bits.  The x coordinate of every copy has
// to be a multiple of 4 (16 bytes): element tiles of weight gradients start at multiples of 16, all other boxes at multiples of their columns.
inline CUtensorMap boxMap(const void *data, int rows, int cols, CUtensorMapSwizzle swizzle, int boxCols = kBoxCols, int boxRows = kBoxRows) {
    CUtensorMap map;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(cols) * 4};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(boxCols), static_cast<cuuint32_t>(boxRows)};
    const cuuint32_t elementStrides[2] = {1, 1};
    const CUresult rc = encodeTiled()(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void *>(data), dims, strides, box, elementStrides,
                                      CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (rc != CUDA_SUCCESS) fail(RXMET_ERR_CUDA, "cuTensorMapEncodeTiled failed with %d", static_cast<int>(rc));
    return map;
}

#ifdef __CUDACC__
// One box to shared memory; completes on `bar`.
__device__ __forceinline__ void copyBox(uint32_t to, const CUtensorMap *map, int col, int row, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(to), "l"(map), "r"(col),
                 "r"(row), "r"(bar)
                 : "memory");
}
#endif

}  // namespace rxmet
