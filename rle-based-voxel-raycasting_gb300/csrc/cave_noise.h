// The generator's simplex noise (gen::simplex3) without integer conversions,
// integer divisions or branches: the same float operations in the same order,
// so the same bits, for non-negative coordinates below kCaveCoordLimit.
//
//  - floor(v) is v + 2^23 - 2^23 lowered by one where it came out above v; the
//    sum's low mantissa bits are the integer.  i + j + k is exact in floats.
//  - The six orders of (x0, y0, z0) are three comparisons a, b, c.
//  - A gradient is two of the three axes with signs; the axis with factor 0
//    adds a zero, which changes no sum here: n starts at +0 and x + (+-0) = x.
//    The table holds the pair and the signs of perm[i] % 12 as bits.
//  - A corner out of reach adds w = 0 instead of being skipped, likewise.
#pragma once

#include <cstdint>

#include "exact_steps.h"
#include "scenegen_math.h"

namespace rle {
namespace gen {

constexpr float kCaveCoordLimit = 1048576.0f;  // 2^20: every sum below stays under 2^22

// Bits of the gradient of hash h: sign of the first axis (31), of the second
// (30), the first axis is y (1), the second axis is y (0).
RLE_HD uint32_t grad_code(int h) {
    const int e = h % 12, pair = e >> 2;
    return (e & 1 ? 0x80000000u : 0u) | (e & 2 ? 0x40000000u : 0u) | (pair == 2 ? 2u : 0u) | (pair == 0 ? 1u : 0u);
}

// Floor of 0 <= v < 2^22; *low its low eight bits.
RLE_HD float floor_low(float v, int* low) {
    const float m = 8388608.0f;
    float up = v + m;
    float f = up - m;
    if (f > v) {
        f -= 1.0f;
        up -= 1.0f;
    }
    *low = static_cast<int>(bits_of(up) & 255u);
    return f;
}

// One corner at (x, y, z) from the point, its gradient `code`.
RLE_HD float corner(float n, uint32_t code, float x, float y, float z) {
    float w = 0.6f - x * x - y * y - z * z;
    w = w > 0.0f ? w : 0.0f;
    const float u = code & 2u ? y : x, v = code & 1u ? y : z;
    const float g = float_of(bits_of(u) ^ (code & 0x80000000u)) + float_of(bits_of(v) ^ ((code << 1) & 0x80000000u));
    w *= w;
    return n + w * w * g;
}

// simplex3 at (x, y, z); perm and code are indexed 0..511 (code[i] =
// grad_code(perm[i])).
RLE_HD float cave_simplex(const uint8_t* perm, const uint32_t* code, float x, float y, float z) {
    const float F = 1.0f / 3.0f, G = 1.0f / 6.0f;
    const float s = (x + y + z) * F;
    int ii, jj, kk;
    const float i = floor_low(x + s, &ii), j = floor_low(y + s, &jj), k = floor_low(z + s, &kk);
    const float t = (i + j + k) * G;
    const float x0 = x - (i - t), y0 = y - (j - t), z0 = z - (k - t);
    const bool a = x0 >= y0, b = y0 >= z0, c = x0 >= z0;
    const bool i1 = a && c, j1 = !a && b, k1 = !i1 && !j1;
    const bool i2 = a || c, j2 = !a || b, k2 = !(b && c);
    const int p0 = perm[kk], p1 = perm[kk + 1];
    const uint32_t h0 = code[ii + perm[jj + p0]];
    const uint32_t h1 = code[ii + (i1 ? 1 : 0) + perm[jj + (j1 ? 1 : 0) + (k1 ? p1 : p0)]];
    const uint32_t h2 = code[ii + (i2 ? 1 : 0) + perm[jj + (j2 ? 1 : 0) + (k2 ? p1 : p0)]];
    const uint32_t h3 = code[ii + 1 + perm[jj + 1 + p1]];
    float n = corner(0.0f, h0, x0, y0, z0);
    n = corner(n, h1, x0 - (i1 ? 1.0f : 0.0f) + G, y0 - (j1 ? 1.0f : 0.0f) + G, z0 - (k1 ? 1.0f : 0.0f) + G);
    n = corner(n, h2, x0 - (i2 ? 1.0f : 0.0f) + 2.0f * G, y0 - (j2 ? 1.0f : 0.0f) + 2.0f * G,
               z0 - (k2 ? 1.0f : 0.0f) + 2.0f * G);
    n = corner(n, h3, x0 - 1.0f + 3.0f * G, y0 - 1.0f + 3.0f * G, z0 - 1.0f + 3.0f * G);
    return 32.0f * n;
}

// gen::carved for coordinates below the limit; inv = 1 / cave_period.
RLE_HD bool cave_carved(const Consts& p, const uint8_t* perm, const uint32_t* code, float inv, int x, int y, int z) {
    const float fx = static_cast<float>(x) * inv, fy = static_cast<float>(y) * inv * 4.0f,
                fz = static_cast<float>(z) * inv;
    const float d = cave_simplex(perm, code, fx, fy, fz) +
                    0.5f * cave_simplex(perm, code, 2.0f * fx + 17.0f, 2.0f * fy, 2.0f * fz + 31.0f);
    return d > p.cave_threshold;
}

// Whether every noise coordinate of the grid is within the limit (a period so
// short that it is not takes gen::carved, whose floors saturate).
RLE_HD bool cave_coords_fit(const Consts& p) {
    const double inv = static_cast<double>(1.0f / p.cave_period);
    return (8.0 * p.sy + 2.0 * p.sx + 2.0 * p.sz) * inv + 64.0 < static_cast<double>(kCaveCoordLimit);
}

}  // namespace gen
}  // namespace rle
