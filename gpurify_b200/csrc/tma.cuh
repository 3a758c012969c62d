// TMA tile loads (cp.async.bulk.tensor) of FP32 matrices into
// the 128-byte-swizzled layout the tcgen05 shared-memory descriptors name.
#pragma once
#include <cuda.h>

#include "gpx_common.h"

namespace gpx {

// Map of a row-major rows x ld FP32 matrix (ld a multiple of 32, base on 16
// bytes) as ld / 32 column atoms (one 128-byte swizzle atom per row), loaded in
// tiles of box_rows rows x `atoms` atoms, atom-major.  Rows past the end read
// as zero.  A tile starts at an atom's first column, on 128 bytes.
inline CUtensorMap tma_map_f32(const float* base, int64_t rows, int ld, int box_rows, int atoms) {
    using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult found;
        GPX_CUDA(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &found));
        if (found != cudaDriverEntryPointSuccess) throw Error(GPX_ERR_CUDA, "cuTensorMapEncodeTiled not available");
        return reinterpret_cast<Encode>(fn);
    }();
    CUtensorMap m;
    const cuuint64_t dims[3] = {32, (cuuint64_t)rows, (cuuint64_t)ld / 32};
    const cuuint64_t strides[2] = {(cuuint64_t)ld * sizeof(float), 32 * sizeof(float)};
    const cuuint32_t box[3] = {32, (cuuint32_t)box_rows, (cuuint32_t)atoms}, one[3] = {1, 1, 1};
    if (encode(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(base), dims, strides, box, one,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        throw Error(GPX_ERR_INTERNAL, "tensor map refused");
    return m;
}

// Tile of the map from column atom `atom` and row `row` into shared memory at
// dst (on 1024 bytes); its bytes count towards bar.
__device__ __forceinline__ void tma_load_atoms(uint32_t dst, const CUtensorMap* map, int atom, int row, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(dst),
        "l"(map), "r"(0), "r"(row), "r"(atom), "r"(bar)
        : "memory");
}

__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

}  // namespace gpx
