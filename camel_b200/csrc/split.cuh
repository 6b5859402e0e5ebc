// Splitting float32 values into TF32 terms for the 3xTF32 contractions.
#pragma once

#include <cstdint>

namespace ct {

__device__ __forceinline__ float to_tf32(float v) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
    return __uint_as_float(r);
}

// v = hi + lo up to ~2^-22 |v|: hi is v rounded to TF32 (10 explicit mantissa bits), lo the
// TF32 rounding of the exact remainder.
__device__ __forceinline__ void split_tf32(float v, float &hi, float &lo) {
    hi = to_tf32(v);
    if (!isfinite(hi)) {
        if (!isfinite(v)) { // inf / NaN: carried by hi alone
            lo = 0.0f;
            return;
        }
        hi = __uint_as_float(__float_as_uint(v) & 0xFFFFE000u); // rounding overflowed: truncate
    }
    lo = to_tf32(v - hi); // v - hi is exact in float32
}

// The same split without a branch, for code that splits many values per thread and wants their
// dependency chains interleaved (a branch per value serialises them).  Rounding to TF32 (nearest,
// ties away from zero) is an integer operation on the bit pattern: add half a TF32 unit to the
// magnitude, clear the 13 low bits; the carry takes care of the exponent.  Same results as
// split_tf32 for every finite input; an infinity or NaN is carried by hi alone as there.
__device__ __forceinline__ void split_tf32_flat(float v, float &hi, float &lo) {
    const uint32_t u      = __float_as_uint(v);
    const bool v_special  = (u & 0x7f800000u) == 0x7f800000u;           // inf or NaN
    uint32_t h            = (u + 0x1000u) & 0xffffe000u;
    const bool h_overflow = (h & 0x7f800000u) == 0x7f800000u;           // rounding reached the top exponent
    h  = h_overflow ? (u & 0xffffe000u) : h;                            // finite v: truncate instead
    h  = v_special ? u : h;
    hi = __uint_as_float(h);
    const float d    = v - hi;                                          // exact for finite v
    const uint32_t l = (__float_as_uint(d) + 0x1000u) & 0xffffe000u;
    lo = __uint_as_float(v_special ? 0u : l);
}

// A 64 x 64 block of in [k][n] at (k0, n0) into shared memory, by 256 threads, zeros outside: rows of 256 contiguous bytes,
// four 16-byte loads to a thread in flight where the rows are aligned (vec_ok).
__device__ __forceinline__ void transpose_load(
    float (&tile)[64][65], const float *__restrict__ in, int64_t k, int64_t n, int64_t k0, int64_t n0, int vec_ok) {
    if (vec_ok) {
        const int c = (threadIdx.x & 15) * 4, r = threadIdx.x >> 4;
        float4 v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            v[j] = k0 + r + 16 * j < k && n0 + c < n ? __ldcs(reinterpret_cast<const float4 *>(in + (k0 + r + 16 * j) * n + n0 + c))
                                                     : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float *dst = &tile[r + 16 * j][c];
            dst[0] = v[j].x, dst[1] = v[j].y, dst[2] = v[j].z, dst[3] = v[j].w;
        }
    } else {
        const int c = threadIdx.x & 63, r = threadIdx.x >> 6;
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j)
            v[j] = k0 + r + 4 * j < k && n0 + c < n ? __ldcs(in + (k0 + r + 4 * j) * n + n0 + c) : 0.0f;
#pragma unroll
        for (int j = 0; j < 16; ++j)
            tile[r + 4 * j][c] = v[j];
    }
}

} // namespace ct
