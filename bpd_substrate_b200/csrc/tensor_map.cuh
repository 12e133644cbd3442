// Descriptors of the tiled bulk copies of bf16 operands.
#pragma once
#include "bpdq_common.cuh"

#include <cuda.h>
#include <cuda_bf16.h>

namespace bpdq {

// bf16 [..][rows][cols] in boxes of 64 columns (x), box_rows rows and, of three dimensions, box_outer of the outermost, in the 128-byte swizzle;
// ld: elements between rows, ld_outer: between the outermost.  Columns and rows beyond the end read as zeros.
static int bf16_map(CUtensorMap* map, const void* p, int cols, int rows, long ld, int box_rows, int outer = 0, long ld_outer = 0, int box_outer = 0)
{
    typedef CUresult (*TensorMapEncode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                        const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                        CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static TensorMapEncode encode = nullptr;
    if (!encode) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q);
        if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !fn) return latch(BPDQ_ERR_CUDA);
        encode = (TensorMapEncode)fn;
    }
    const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)outer}, strides[2] = {(cuuint64_t)ld * 2, (cuuint64_t)ld_outer * 2};
    const cuuint32_t box[3] = {64, (cuuint32_t)box_rows, (cuuint32_t)box_outer}, estr[3] = {1, 1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, outer ? 3 : 2, const_cast<void*>(p), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : latch(BPDQ_ERR_CUDA - 900 - (int)r);
}

}  // namespace bpdq
