// Host-side helper: the driver's tensor-map encoder (cuTensorMapEncodeTiled), looked up through
// the runtime so that the library does not link against libcuda directly.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace nvfp4 {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static inline EncodeTiledFn encode_tiled_fn() {
    // (a first call waits for another thread's: it must not find "looked up" and nothing yet)
    static const EncodeTiledFn fn = []() -> EncodeTiledFn {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) ==
                cudaSuccess && qres == cudaDriverEntryPointSuccess)
            return (EncodeTiledFn)p;
        return nullptr;
    }();
    return fn;
}

// A matrix of `rows` rows of `inner` elements, `pitch` bytes apart, as boxes of box_rows x box_inner; what lies outside is
// read as zero and not written.
static inline bool tile_map(EncodeTiledFn enc, CUtensorMap* map, CUtensorMapDataType type, const void* base, long long inner,
                            long long rows, long long pitch, int box_inner, int box_rows, CUtensorMapSwizzle swizzle,
                            CUtensorMapL2promotion promotion) {
    const cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)pitch};
    const cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_rows}, estr[2] = {1, 1};
    return enc(map, type, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
               promotion, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// Stages of 256 k: packed bytes [rows][K / 2] in 128-byte swizzled boxes of 128, scale bytes [rows][K / 16] in boxes of 16.
static inline bool packed_map(EncodeTiledFn enc, CUtensorMap* map, const void* base, int rows, int K, int box_rows,
                              CUtensorMapL2promotion promotion) {
    return tile_map(enc, map, CU_TENSOR_MAP_DATA_TYPE_UINT8, base, K / 2, rows, K / 2, 128, box_rows,
                    CU_TENSOR_MAP_SWIZZLE_128B, promotion);
}
static inline bool scales_map(EncodeTiledFn enc, CUtensorMap* map, const void* base, int rows, int K, int box_rows,
                              CUtensorMapL2promotion promotion = CU_TENSOR_MAP_L2_PROMOTION_NONE) {
    return tile_map(enc, map, CU_TENSOR_MAP_DATA_TYPE_UINT8, base, K / 16, rows, K / 16, 16, box_rows,
                    CU_TENSOR_MAP_SWIZZLE_NONE, promotion);
}

}  // namespace nvfp4
