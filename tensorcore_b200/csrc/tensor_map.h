// Host-side construction of TMA tensor maps (cuTensorMapEncodeTiled), looked up through the
// runtime so that the library does not link against the driver library.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace tcb {

using TensorMapEncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                       const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                       CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                       CUtensorMapFloatOOBfill);
inline TensorMapEncodeFn tensor_map_encoder() {
    static TensorMapEncodeFn encode = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            fn = nullptr;
        return reinterpret_cast<TensorMapEncodeFn>(fn);
    }();
    return encode;
}

// Tiled map over a row-major byte matrix [rows][row_bytes] (row_bytes a multiple of 16, base
// 16-byte aligned) with a box of box_rows x box_bytes (box_bytes a multiple of 16).  The matrix is
// described in elements of elem_bytes (1 or 4) because a box is limited to 256 elements per
// dimension: box_bytes / elem_bytes <= 256, box_rows <= 256; the load's x coordinate is in
// elements.  No swizzle, no interleave; parts of a box outside the matrix read as zeros.
inline bool encode_bytes_2d(CUtensorMap* map, const void* base, uint64_t rows, uint64_t row_bytes,
                            uint32_t box_bytes, uint32_t box_rows, uint32_t elem_bytes = 1) {
    const TensorMapEncodeFn encode = tensor_map_encoder();
    if (!encode) return false;
    if (elem_bytes != 1 && elem_bytes != 4) return false;
    if (row_bytes % elem_bytes || box_bytes % elem_bytes) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(row_bytes / elem_bytes), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(row_bytes)};
    const cuuint32_t box[2] = {box_bytes / elem_bytes, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return encode(map, elem_bytes == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// fp16 matrix [rows][cols], cols a multiple of 64, base 16-byte aligned, as [cols / 64] slices of 128-byte
// rows written to shared memory with the 128-byte swizzle: one load at (0, row, slice) brings
// box_slices consecutive K slices of box_rows rows, slice after slice.  Rows outside read as zeros.
inline bool encode_f16_slices_sw128(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols,
                                    uint32_t box_rows, uint32_t box_slices) {
    const TensorMapEncodeFn encode = tensor_map_encoder();
    if (!encode || cols % 64 || box_rows > 256) return false;
    const cuuint64_t dims[3] = {64, static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(cols / 64)};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(cols * 2), 128};
    const cuuint32_t box[3] = {64, box_rows, box_slices};
    const cuuint32_t estr[3] = {1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Row-major 16-bit matrix [rows][cols] (leading dimension ld, a multiple of 8) with a box of box_rows x 64
// elements (128 bytes), written to shared memory with the 128-byte swizzle.  Parts outside read as zeros.
inline bool encode_rows_sw128(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows) {
    const TensorMapEncodeFn encode = tensor_map_encoder();
    if (!encode || ld % 8) return false;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {ld * 2};
    const cuuint32_t box[2] = {64, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// fp16 [heads][rows][cols] as boxes of box_rows x 64 elements of one head, written to shared memory with the
// 128-byte swizzle: a load at (64 * slab, row, head).  Rows past the head's end read as zeros.
inline bool encode_heads_sw128(CUtensorMap* map, const void* base, uint64_t heads, uint64_t rows, uint64_t cols, uint32_t box_rows) {
    const TensorMapEncodeFn encode = tensor_map_encoder();
    if (!encode || cols % 64 || box_rows > 256) return false;
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(heads)};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(cols * 2), static_cast<cuuint64_t>(rows * cols * 2)};
    const cuuint32_t box[3] = {64, box_rows, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace tcb
