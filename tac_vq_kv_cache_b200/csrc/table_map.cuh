// Tensor maps over codeword tables, for kernels that fetch whole tables with TMA copies.
#pragma once

#include <cstring>

#include <cuda.h>  // CUtensorMap and the driver's encoder signature; the entry point is looked up at run time

#include "common.cuh"

namespace tacvq {

// cuTensorMapEncodeTiled, looked up through the runtime so that the library does not link against the driver
typedef CUresult (*TensorMapEncoder)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                     const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                     CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline TensorMapEncoder tensor_map_encoder() {
    static const TensorMapEncoder found = [] {
        void *entry = nullptr;
        cudaDriverEntryPointQueryResult status;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &entry, cudaEnableDefault, &status) != cudaSuccess ||
            status != cudaDriverEntryPointSuccess)
            entry = nullptr;
        return reinterpret_cast<TensorMapEncoder>(entry);
    }();
    return found;
}

// The fp16 tables as a 2-D tensor [all words][d] read in boxes of 256 words x 64 elements with the 128-byte swizzle.
// (d = 32: boxes of 256 x 32 with the 64-byte swizzle).  Returns 0 when no map could be made.
inline int make_table_map(CUtensorMap *map, const void *tables, int64_t words, int d) {
    memset(map, 0, sizeof(*map));
    const TensorMapEncoder encode = tensor_map_encoder();
    if (encode == nullptr || words < kMaxWords) return 0;
    const cuuint64_t dims[2] = {(cuuint64_t)d, (cuuint64_t)words};
    const cuuint64_t strides[1] = {(cuuint64_t)d * 2};
    const cuuint32_t box[2] = {(cuuint32_t)(d < 64 ? d : 64), (cuuint32_t)kMaxWords};
    const cuuint32_t steps[2] = {1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void *>(tables), dims, strides, box, steps,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, d < 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 1 : 0;
}

}  // namespace tacvq
