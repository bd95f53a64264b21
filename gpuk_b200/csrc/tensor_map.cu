// Encoding of TMA tensor maps.  The driver's function is looked up through the runtime, so nothing links against libcuda.
#include <cuda.h>
#include <cuda_runtime.h>

#include "tensor_core.cuh"

int gpuk::encode_map(CUtensorMap *map, CUtensorMapDataType type, const void *base, int rank, const uint64_t *sizes, const uint64_t *strides, const uint32_t *box,
                     CUtensorMapSwizzle swizzle) {
    using Encode = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &found) != cudaSuccess || found != cudaDriverEntryPointSuccess)
            fn = nullptr;
        return reinterpret_cast<Encode>(fn);
    }();
    if (!encode) return -1;
    const cuuint32_t ones[5] = {1, 1, 1, 1, 1};
    return static_cast<int>(encode(map, type, static_cast<cuuint32_t>(rank), const_cast<void *>(base), sizes, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                   swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE));
}
