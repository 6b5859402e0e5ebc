// Tensor-map encoding shared by the contraction kernels (the driver entry point is fetched
// through the runtime, so the library carries no link-time dependency on libcuda).
#pragma once

#include "common.cuh"

#include <cuda.h>

namespace ct {

// A tiled float32 tensor map of `rank` dimensions (innermost first): extents `dims`, byte strides
// of dimensions 1.. in `strides` (rank - 1 entries), box extents `box`, the 128- or 64-byte
// swizzle (0: none), out-of-range elements read as zero.
ct_status encode_tiled_map_f32(
    CUtensorMap *map, const void *base, int rank, const uint64_t *dims, const uint64_t *strides, const uint32_t *box,
    int swizzle_bytes);
// The same for float16 elements.
ct_status encode_tiled_map_f16(
    CUtensorMap *map, const void *base, int rank, const uint64_t *dims, const uint64_t *strides, const uint32_t *box,
    int swizzle_bytes);

// conv2d with the filters in tensor memory (conv_tmem.cu).
bool conv_tmem_applicable(int64_t c, int64_t h, int64_t w, int64_t ko, int64_t kh, int64_t kw, int64_t stride,
                          int64_t pad, bool *pool_ok = nullptr);
ct_status conv_tmem_filters(
    DeviceState *st, const float *x, const float *w, const float *bias, int64_t batch, int64_t c, int64_t h, int64_t wd,
    int64_t ko, int64_t kh, int64_t kw, int64_t pad, int act, int pool, float *out);

// conv2d with one input halo per tile and channel block serving every tap (conv_halo.cu).
bool conv_halo_applicable(int64_t c_pad, int64_t h, int64_t w, int64_t ko, int64_t kh, int64_t kw, int64_t stride,
                          int64_t pad);
// The float16 planes of an image: sub-images of the rows (columns) that are alike modulo row_mod (col_mod), a bit of `used`
// for each that is needed; the others have no place in the planes.  tf32_plain: tf32 planes are not taken apart.
struct ConvSubImages {
    int row_mod = 1, col_mod = 1;
    uint32_t used = 1;
    bool tf32_plain = false;
    int rows = 0, cols = 0; // of a sub-image
    int y0 = 0, x0 = 0;     // the input's row and column that row 0 and column 0 of the first one are
};
int conv_range_slices(int64_t batch, int64_t count);
ct_status conv_prepass(
    const float *x, const float *w, int64_t batch, int64_t c, int64_t h, int64_t wd, int64_t c_pad, int64_t ko, int64_t taps,
    void *filters16, void *filters32, size_t plane16, size_t plane32, const uint8_t *order, float *filter_scale, const float *bias, float *bias_copy,
    void *ranges, float *image_scale, void *slots, const ConvSubImages &sub);
// x NCHW and w OIHW float32; c_pad: channels rounded up to 32.
ct_status conv_halo(
    DeviceState *st, const float *x, const float *w, int64_t batch, int64_t c, int64_t c_pad, int64_t h, int64_t wd, int64_t ko,
    int64_t kh, int64_t kw, int64_t stride, int64_t pad, const float *bias, int act, float *out);

} // namespace ct
