// Host-side creation of TMA tensor maps through the driver entry point (no link-time
// dependency on libcuda). Maps describe plain row-major byte matrices [rows][row_bytes]
// loaded as boxes of [box_rows][row_bytes] with the 128-byte shared-memory swizzle.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

namespace rivoli {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled_fn() {
    static std::atomic<EncodeTiledFn> known{nullptr};
    EncodeTiledFn fn = known.load(std::memory_order_relaxed);
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess) {
            fn = reinterpret_cast<EncodeTiledFn>(p);
            known.store(fn, std::memory_order_relaxed);
        }
    }
    return fn;
}

// rows x row_bytes bytes (row_bytes == 128 here: one swizzle row), box = box_rows full rows.
// Returns 0, or 1008 if the driver refuses.
inline int make_tmap_rows_sw128(CUtensorMap* out, const void* base, uint64_t rows, uint32_t row_bytes,
                                uint32_t box_rows) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return 1008;
    const cuuint64_t dims[2] = {row_bytes, rows};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {row_bytes, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : 1008;
}

}  // namespace rivoli
