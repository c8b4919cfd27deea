// tma_map.h -- host side of the TMA tensor maps: cuTensorMapEncodeTiled taken
// from the driver at run time (no link against libcuda) and the 2D maps that
// the tensor-core kernels load through.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include "../../include/qlpix.h"

namespace qlpix {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn get_encode()
{
    static const EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return (EncodeTiledFn)p;
        return (EncodeTiledFn) nullptr;
    }();
    return fn;
}

// A row-major [rows][cols] array of F16 or FP32, boxes of box_rows x
// box_cols; the swizzle spans one box row (128 or 64 bytes).
inline int make_map_box(CUtensorMap* map, void* base, size_t rows, size_t cols, bool half, int box_rows, int box_cols)
{
    EncodeTiledFn enc = get_encode();
    if (!enc) return QLP_ERR_CUDA;
    const size_t esz = half ? 2 : 4;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * esz};
    cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    const CUtensorMapSwizzle sw = (box_cols * esz == 64) ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B;
    CUresult r = enc(map, half ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, base, dims,
                     strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? QLP_OK : QLP_ERR_CUDA;
}

}  // namespace qlpix
