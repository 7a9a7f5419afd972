// Tensor maps for TMA tensor copies: the driver's encoder, looked up once.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace gf {

// Row-major tensor of `rank` dimensions (innermost first; strides in bytes of dimensions 1..), 128-byte swizzle or none, zero fill.
inline int encode_map(CUtensorMap *map, CUtensorMapDataType type, int rank, void *base, const uint64_t *dims, const uint64_t *strides,
                      const uint32_t *box, const char *what, bool swizzle = true) {
    typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                      const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                      CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        GF_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
        GF_REQUIRE(p != nullptr && q == cudaDriverEntryPointSuccess, "cuTensorMapEncodeTiled is not available in this driver");
        fn = (EncodeTiledFn)p;
    }
    cuuint64_t d[5], st[4];
    cuuint32_t b[5], one[5];
    for (int i = 0; i < rank; ++i) { d[i] = dims[i]; b[i] = box[i]; one[i] = 1; if (i) st[i - 1] = strides[i - 1]; }
    const CUresult r = fn(map, type, rank, base, d, st, b, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    GF_REQUIRE(r == CUDA_SUCCESS, std::string("cuTensorMapEncodeTiled failed for the ") + what + ": " + std::to_string((int)r));
    return 0;
}

}  // namespace gf
