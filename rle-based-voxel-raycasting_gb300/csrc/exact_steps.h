// Chains of single-precision additions, x + g + g + ..., rounded after every
// step, without taking the steps.
//
// The DDA and the fill accumulate their values step by step, as the reference
// does, and every pixel depends on the rounding.  While the sums stay in one
// binade they are multiples of one ulp, and adding g adds g rounded to that
// ulp: the same multiple at every step, except that where g lies half way
// between two multiples the tie goes to the even sum -- which holds from the
// first such step on, so that two equal steps in a row settle it.  n steps
// from a sum x are then x + n * step; that is a multiple of the ulp inside the
// binade, so a fused multiply-add gives it exactly.  The sums being monotone,
// it is enough that the first and the last lie in the binade.  Where the
// magnitude falls, a last sum of exactly 2^e does not count: just below 2^e
// the ulp is half as large, and the true sum may not have been rounded up.
//
// Compiled by nvcc for the kernels and by the host compiler for the tests.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define RLE_STEP_FN __host__ __device__ __forceinline__
#else
#define RLE_STEP_FN inline
#endif

namespace rle {

RLE_STEP_FN uint32_t bits_of(float f) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(f);
#else
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return u;
#endif
}
RLE_STEP_FN float float_of(uint32_t u) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float f;
    std::memcpy(&f, &u, 4);
    return f;
#endif
}

// The last sum v lies in the binade of the first, a, in whichever direction
// the sums run (a zero mantissa is left out in both).
RLE_STEP_FN bool in_binade(float a, float v) {
    return ((bits_of(a) ^ bits_of(v)) & 0xff800000u) == 0u && (bits_of(v) & 0x007fffffu) != 0u;
}

// Whether the n sums after x are x + step, x + 2 * step, ... exactly; *step is
// g rounded to the ulp of x.
RLE_STEP_FN bool steady_step(float x, float g, int n, float* step) {
    const float x1 = x + g, d = x1 - x;
    *step = d;
    return (x1 + g) - x1 == d && in_binade(x, fmaf(static_cast<float>(n), d, x));
}

// The sum after m steps.
RLE_STEP_FN float accumulate(float x, float g, int m) {
    while (m > 0) {
        const float x1 = x + g, x2 = x1 + g;
        if (m == 1) return x1;
        // inf and NaN stay what they are two steps on
        if (m == 2 || (bits_of(x1) & 0x7f800000u) == 0x7f800000u) return x2;
        const float d = (x2 + g) - x2;
        if (d == 0.0f) return x2;
        const float v = fmaf(static_cast<float>(m - 2), d, x2);
        if (in_binade(x1, v)) return v;
        // to about the end of x1's binade: any count that stays in it will do
        const float edge = float_of((bits_of(x1) & 0xff800000u) + (fabsf(x2) > fabsf(x1) ? 0x00800000u : 0u));
#ifdef __CUDA_ARCH__
        const float room = __fdividef(edge - x2, d) - 1.0f;
#else
        const float room = (edge - x2) / d - 1.0f;
#endif
        const int n = room >= 1.0f ? (room < static_cast<float>(m - 2) ? static_cast<int>(room) : m - 2) : 0;
        const float w = fmaf(static_cast<float>(n), d, x2);
        const bool in = in_binade(x1, w);
        x = in ? w : x2;
        m -= 2 + (in ? n : 0);
    }
    return x;
}

}  // namespace rle
