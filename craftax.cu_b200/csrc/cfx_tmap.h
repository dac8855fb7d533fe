// Functions of the driver through their entry points (no link-time dependency on libcuda), and the
// host-side construction of TMA tensor maps.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cstdint>

namespace cfx {

typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                    const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                    const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                    CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// A function of the driver, or NULL
inline void* driver_entry(const char* name) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    return cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess ? p : nullptr;
}

inline PFN_encodeTiled get_encode_tiled() {
    static PFN_encodeTiled fn = nullptr;
    if (!fn) fn = (PFN_encodeTiled)driver_entry("cuTensorMapEncodeTiled");
    return fn;
}

// 2-D row-major tensor [rows][cols] of `elem_bytes`-wide elements with a row pitch of
// `pitch_bytes` (multiple of 16); box = [box_rows][box_cols].  Returns false on failure.
inline bool make_tmap_2d(CUtensorMap* map, CUtensorMapDataType dt, int elem_bytes, void* base,
                         uint64_t rows, uint64_t cols, uint64_t pitch_bytes, uint32_t box_rows,
                         uint32_t box_cols, CUtensorMapSwizzle swz) {
    PFN_encodeTiled enc = get_encode_tiled();
    if (!enc) return false;
    (void)elem_bytes;
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {pitch_bytes};
    cuuint32_t box[2] = {box_cols, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, dt, 2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

// Blocks of rows of 64 16-bit elements (128 bytes), all contiguous: [blocks][rows][64]; box = [box_blocks][box_rows][64].
inline bool make_tmap_blocks(CUtensorMap* map, void* base, uint64_t blocks, uint64_t rows, uint32_t box_blocks, uint32_t box_rows) {
    PFN_encodeTiled enc = get_encode_tiled();
    if (!enc) return false;
    cuuint64_t dims[3] = {64, rows, blocks};
    cuuint64_t strides[2] = {128, rows * 128};
    cuuint32_t box[3] = {64, box_rows, box_blocks};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

// Groups of parts of rows of 64 16-bit elements (128 bytes), all contiguous: [groups][parts][rows][64]; box =
// [box_groups][box_parts][rows][64].
inline bool make_tmap_parts(CUtensorMap* map, void* base, uint64_t groups, uint64_t parts, uint64_t rows, uint32_t box_groups,
                            uint32_t box_parts) {
    PFN_encodeTiled enc = get_encode_tiled();
    if (!enc) return false;
    cuuint64_t dims[4] = {64, rows, parts, groups};
    cuuint64_t strides[3] = {128, rows * 128, parts * rows * 128};
    cuuint32_t box[4] = {64, (cuuint32_t)rows, box_parts, box_groups};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 4, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

}  // namespace cfx
