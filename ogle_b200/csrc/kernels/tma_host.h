// Host-side TMA descriptor helpers shared by the kernels that use tensor maps.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace ogle {

// Address of the library's device status word on the current device.
int* error_flag_ptr();

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

typedef CUresult (*EncodeIm2colFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const int*, const int*, cuuint32_t, cuuint32_t, const cuuint32_t*,
                                   CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline void* driver_entry(const char* name) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) p = nullptr;
    return p;
}
inline EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = reinterpret_cast<EncodeTiledFn>(driver_entry("cuTensorMapEncodeTiled"));
    return fn;
}
inline EncodeIm2colFn encode_im2col_fn() {
    static EncodeIm2colFn fn = reinterpret_cast<EncodeIm2colFn>(driver_entry("cuTensorMapEncodeIm2col"));
    return fn;
}

// swizzle: CU_TENSOR_MAP_SWIZZLE_128B for UMMA operand tiles, _NONE for plain tiles.
inline bool make_map_sw(CUtensorMapSwizzle swizzle, CUtensorMap* m, const void* ptr, int rank, const cuuint64_t* dims, const cuuint64_t* strides_bytes,
              const cuuint32_t* box, const cuuint32_t* estr) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, (cuuint32_t)rank, const_cast<void*>(ptr), dims, strides_bytes,
                    box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}


inline bool make_map(CUtensorMap* m, const void* ptr, int rank, const cuuint64_t* dims, const cuuint64_t* strides_bytes,
                     const cuuint32_t* box, const cuuint32_t* estr) {
    return make_map_sw(CU_TENSOR_MAP_SWIZZLE_128B, m, ptr, rank, dims, strides_bytes, box, estr);
}

// Map of an image tensor of 16-byte pixels [n][h][w] whose boxes take `cols` pixels of `rows` rows. A pixel is two 8-byte
// elements of one row-long extent, not an extent of its own: the copy engine takes a row of a box as a whole instead of
// pixel by pixel. At most 128 columns; coordinates (2 * column, row, image, 0).
inline bool make_map_pixels(CUtensorMap* m, const void* ptr, int W, int H, int N, int cols, int rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)W * 2, (cuuint64_t)H, (cuuint64_t)N, 1};
    const cuuint64_t str[3] = {(cuuint64_t)W * 16, (cuuint64_t)W * 16 * H, (cuuint64_t)W * 16 * H * N};
    const cuuint32_t box[4] = {(cuuint32_t)cols * 2, (cuuint32_t)rows, 1, 1}, es[4] = {1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, const_cast<void*>(ptr), dims, str, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// im2col map of an activation tensor [n][h][w][c] (dims and strides channel first, as above): a copy takes `channels` of
// `pixels` consecutive positions of the window's first tap, which walk the image from `lower` to its far edge plus `upper`
// ({w, h} each), row after row and image after image; positions outside the image read zero.
inline bool make_map_im2col(CUtensorMap* m, const void* ptr, const cuuint64_t* dims, const cuuint64_t* strides_bytes,
                            const int* lower, const int* upper, int channels, int pixels, int stride = 1) {
    EncodeIm2colFn fn = encode_im2col_fn();
    if (!fn) return false;
    const cuuint32_t es[4] = {1, (cuuint32_t)stride, (cuuint32_t)stride, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<void*>(ptr), dims, strides_bytes, lower, upper, (cuuint32_t)channels,
              (cuuint32_t)pixels, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace ogle
