// Splitting float32 matrices into scaled float16 pairs for the tensor-core contractions.
//
// A float32 value is carried as two 11-bit significands, as in the 3xTF32 split (split.cuh), but in
// float16, whose MMAs take 16 values of k in the time a tf32 MMA takes 8 and whose planes are half as
// large.  float16's five exponent bits are made up for by an exact power of two per row of the left
// operand and per column of the right one (the row's largest magnitude is moved to [2^14, 2^15)) and by
// storing the low term 2^11 times larger:
//     v * 2^(14-e) = hi + lo * 2^-11,   hi = half(v * 2^(14-e)),   lo = half((v * 2^(14-e) - hi) * 2^11)
// The pair holds a scaled value to an absolute error of 2^-36 at worst (lo's quantum is then 2^-24) and to 2^-23
// of itself from 2^-13 up, which is what a pair of tf32 terms holds of any value; from 2^-12 up the two terms are the
// same two 11-bit numbers whatever the scale (every bit of lo lies above float16's smallest).
//
// Values below that are exceptions (2^-27 of their row's largest, or less): hi would be subnormal, lo more than 2^-11 of
// it, and the product of two low terms, which no MMA computes, no longer negligible.  Matrices of ordinary values have
// a few per hundred million, so the pre-pass stores zeros for them, lists up to kHalfExceptions of a product, marks
// their rows by the sign of the scale, and the product's epilogue adds value . other operand to the outputs of
// those rows and columns.  A matrix with more of them, or with a row whose exponent is beyond +-60, is computed from
// tf32 planes instead (same launch sequence, no host involvement).  Convolutions, but those through patches, decide
// that per image (and per layer for its filters), see half_range_fits.
#pragma once

#include <cuda_fp16.h>

#include <cstdint>

namespace ct {

constexpr int kHalfLoBits       = 11;
constexpr float kHalfLoScale    = 2048.0f;              // 2^11
constexpr float kHalfLoInv      = 1.0f / 2048.0f;
constexpr float kHalfSmallest   = 1.0f / (1u << 13);    // scaled magnitudes below this are exceptions
constexpr int kHalfMaxExponent  = 60;

struct HalfException {
    int line, k; // 2 * row of the planes + operand (0 left, 1 right), position in the row
    float value; // the planes hold 0 there
};
constexpr int kHalfExceptions = 32;
struct alignas(8) HalfExceptions {
    uint32_t wide;  // a row's exponent does not fit
    uint32_t count; // exceptions found; more than the list holds: the operands need tf32 planes
    HalfException e[kHalfExceptions];
};

// magnitude bits of a finite value, 0 for infinities and NaN (they are carried by hi alone)
__device__ __forceinline__ uint32_t finite_magnitude(float v) {
    const uint32_t u = __float_as_uint(v) & 0x7fffffffu;
    return u < 0x7f800000u ? u : 0u;
}

__device__ __forceinline__ float exact_pow2(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }

// From the largest magnitude of a row: the factor that brings it to [2^14, 2^15) and its inverse.
// False when the exponent is beyond what the float16 form takes.
__device__ __forceinline__ bool half_scale(uint32_t max_bits, float &scale, float &inverse) {
    int e = max_bits == 0 ? 14 : (int)(max_bits >> 23) - 127;
    const bool ok = e >= -kHalfMaxExponent && e <= kHalfMaxExponent;
    e       = e < -kHalfMaxExponent ? -kHalfMaxExponent : (e > kHalfMaxExponent ? kHalfMaxExponent : e);
    scale   = exact_pow2(14 - e);
    inverse = exact_pow2(e - 14);
    return ok;
}

// The range of the values that share a scale, gathered with two instructions a value: .x the largest magnitude (an
// infinity or NaN as what it is), .y the smallest non-zero one less 1 (all ones: there is none).
constexpr uint32_t kNoneSmallest = 0xffffffffu;
__device__ __forceinline__ void range_take(uint2 &r, float v) {
    const uint32_t u = __float_as_uint(v) & 0x7fffffffu;
    r.x = max(r.x, u);
    r.y = min(r.y, u - 1u);
}
__device__ __forceinline__ uint2 range_join(uint2 a, uint2 b) { return make_uint2(max(a.x, b.x), min(a.y, b.y)); }
__device__ __forceinline__ uint2 range_warp(uint2 r) {
    return make_uint2(__reduce_max_sync(0xffffffffu, r.x), __reduce_min_sync(0xffffffffu, r.y));
}

// Whether float16 pairs under one scale hold every value of the range as the two 11-bit terms that any other
// scale would give: the rule of the convolutions, whose scales belong to an image or to a tile of it.  An image for
// which this is true has the same bits in its outputs whatever part of it a scale was taken over.
constexpr float kHalfExact = 1.0f / (1u << 12);
__device__ __forceinline__ bool half_range_fits(uint2 r, float &scale, float &inverse) {
    const bool ok = half_scale(r.x, scale, inverse);
    return ok && (r.y == kNoneSmallest || __uint_as_float(r.y + 1u) * scale >= kHalfExact);
}

// The same for a part of an image, by itself: true for every part of an image that fits.  A part may lie wholly below the smallest
// exponent where its image does not (a scale of 2^74 holds all that an image that fits can have, 2^-86 and up), so it has
// that scale and no floor of its own.
__device__ __forceinline__ bool half_tile_fits(uint2 r, float &scale, float &inverse) {
    half_scale(r.x, scale, inverse);
    return r.x < (uint32_t)(kHalfMaxExponent + 128) << 23 && (r.y == kNoneSmallest || __uint_as_float(r.y + 1u) * scale >= kHalfExact);
}

__device__ __forceinline__ bool half_exception(float v, float scale) { return v != 0.0f && fabsf(v * scale) < kHalfSmallest; }

// Returns true, and zeros, for an exception.
__device__ __forceinline__ bool split_half(float v, float scale, __half &hi, __half &lo) {
    const bool exception = half_exception(v, scale);
    v  = exception ? 0.0f : v * scale;
    hi = __float2half_rn(v);
    const float d = (v - __half2float(hi)) * kHalfLoScale; // exact for finite v
    lo = isfinite(v) ? __float2half_rn(d) : __half(0.0f);
    return exception;
}

// Two scaled values of a range that fits (half_range_fits): finite, no exceptions.
__device__ __forceinline__ void split_half_pair(float a, float b, __half2 &hi, __half2 &lo) {
    hi = __floats2half2_rn(a, b);
    lo = __floats2half2_rn(__fmul_rn(__fsub_rn(a, __low2float(hi)), kHalfLoScale), __fmul_rn(__fsub_rn(b, __high2float(hi)), kHalfLoScale));
}

// Whether either operand needs its tf32 planes: one 8-byte load for each list, and one in all where they share it.  As
// four loads in a row they cost an idle launch 3 us, and a second volatile load of the same words 0.8 us.
__device__ __forceinline__ bool half_wide(const HalfExceptions *a, const HalfExceptions *b) {
    const uint64_t va = *reinterpret_cast<const volatile uint64_t *>(a);
    bool wide         = (uint32_t)va != 0u || (uint32_t)(va >> 32) > kHalfExceptions;
    if (a != b) {
        const uint64_t vb = *reinterpret_cast<const volatile uint64_t *>(b);
        wide |= (uint32_t)vb != 0u || (uint32_t)(vb >> 32) > kHalfExceptions;
    }
    return wide;
}

// More exceptions than the list holds: the rest need not be looked for.
__device__ __forceinline__ bool half_overfull(const HalfExceptions *x) {
    return const_cast<const volatile HalfExceptions *>(x)->count > kHalfExceptions;
}

// A whole warp records its lanes' exceptions among the values v; true if there were any.  Once the list is over-full the
// count is left alone: a matrix of nothing else would queue up at one word.
__device__ __forceinline__ bool half_record(HalfExceptions *x, float v, float scale, int operand, int64_t line, int64_t k) {
    const bool mine     = half_exception(v, scale);
    const uint32_t mask = __ballot_sync(0xffffffffu, mine);
    if (mask == 0u)
        return false;
    const int lane = threadIdx.x & 31;
    uint32_t at    = kHalfExceptions;
    if (lane == 0 && !half_overfull(x))
        at = atomicAdd(&x->count, (uint32_t)__popc(mask));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(mask & ((1u << lane) - 1u));
    if (mine && at < kHalfExceptions)
        x->e[at] = HalfException{(int)line * 2 + operand, (int)k, v};
    return true;
}

} // namespace ct
