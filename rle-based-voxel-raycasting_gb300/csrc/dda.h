// The 2D DDA of a column ray (src/Cuda_Render.h:306-416), step by step and
// many steps at once.  Compiled by nvcc for the kernels and by the host
// compiler for the tests.
#pragma once

#include "exact_steps.h"

namespace rle {

// Next event of either axis -- its distance ddA along the ray and its
// intersection (iAx, iAy) -- with their steps, and the event before
// (distance, intersection, axis).
struct Dda {
    float g0x, g0y, g1x, g1y, gd0, gd1;
    float i0x, i0y, i1x, i1y, dd0, dd1;
    float dd_now, pnx, pny;
    int index;
};

// One step (:376-414), written with selects: the chain from one step to the
// next is a compare and a select (the additions for both axes are issued
// beside the compare), shorter than a branch on the compare.
RLE_STEP_FN void dda_step(Dda& d) {
    const bool c1 = d.dd1 < d.dd0;
    d.dd_now = c1 ? d.dd1 : d.dd0;
    d.index = c1 ? 1 : 0;
    d.pnx = c1 ? d.i1x : d.i0x;
    d.pny = c1 ? d.i1y : d.i0y;
    const float n1 = d.dd1 + d.gd1, n0 = d.dd0 + d.gd0;
    const float a1x = d.i1x + d.g1x, a1y = d.i1y + d.g1y;
    const float a0x = d.i0x + d.g0x, a0y = d.i0y + d.g0y;
    d.dd1 = c1 ? n1 : d.dd1;
    d.i1x = c1 ? a1x : d.i1x;
    d.i1y = c1 ? a1y : d.i1y;
    d.dd0 = c1 ? d.dd0 : n0;
    d.i0x = c1 ? d.i0x : a0x;
    d.i0y = c1 ? d.i0y : a0y;
}

// Whether the steps can be skipped over: a ray that runs along an axis to the
// last bit has infinite steps on the other (and NaN where those meet a zero).
RLE_STEP_FN bool dda_can_jump(const Dda& d) { return (d.dd0 + d.gd0) + (d.dd1 + d.gd1) < 1e30f; }

// The steps of the six chains, rounded to the ulp of their binades, as long as
// none leaves its binade.  steadyA: two steps of axis A from here are equal
// (exact_steps.h) and its chains grow in magnitude, so that n steps stay
// between their first and last sums; without it only one step is known.  The
// step along an axis itself (g0x, g1y) is a whole number, hence exact while
// the ulp is at most 1.
struct DdaCache {
    float s0, s1, r0, r1, inv;
    bool steady0, steady1;
};

RLE_STEP_FN DdaCache dda_cache(const Dda& d) {
    DdaCache c;
    const float x0 = d.dd0 + d.gd0, x1 = d.dd1 + d.gd1, y0 = d.i0y + d.g0y, y1 = d.i1x + d.g1x;
    c.s0 = x0 - d.dd0;
    c.s1 = x1 - d.dd1;
    c.r0 = y0 - d.i0y;
    c.r1 = y1 - d.i1x;
    c.steady0 = (x0 + d.gd0) - x0 == c.s0 && (y0 + d.g0y) - y0 == c.r0 && fabsf(d.i0x) < 8388608.0f &&
                (((bits_of(d.i0x) ^ bits_of(d.g0x)) | (bits_of(d.i0y) ^ bits_of(d.g0y))) >> 31) == 0u;
    c.steady1 = (x1 + d.gd1) - x1 == c.s1 && (y1 + d.g1x) - y1 == c.r1 && fabsf(d.i1y) < 8388608.0f &&
                (((bits_of(d.i1x) ^ bits_of(d.g1x)) | (bits_of(d.i1y) ^ bits_of(d.g1y))) >> 31) == 0u;
#ifdef __CUDA_ARCH__
    c.inv = __fdividef(1.0f, c.s0 + c.s1);
#else
    c.inv = 1.0f / (c.s0 + c.s1);
#endif
    return c;
}

// The event of step k from here (0 = the next) and the state after it, without
// the k steps before, bit for bit theirs: the state while `ok`, the event also
// at the first k that is not (for k = 0 always).
//
// The walk merges the events of two axes, each at the distances that a chain
// of additions gives (dd0, dd0 + gd0, ... and dd1, dd1 + gd1, ...): its first
// k steps take n of axis 0 and m = k - n of axis 1, where n is the one count
// with A0[n-1] <= A1[m] and A1[m-1] < A0[n] (equal distances go to axis 0).
// With terms x + n * step that is the floor of a quotient below 100 whose
// error is a few ulp, so rounding it to a whole number by a large addend is
// off by one at most, and checked.  `kept`: the cache holds after step k, too.
struct DdaJump {
    bool axis1, ok, kept;
    float dd, px, py;                   // the event
    float dd0, i0x, i0y, dd1, i1x, i1y;  // the state after it
};

RLE_STEP_FN DdaJump dda_jump(const Dda& d, const DdaCache& c, float kf) {
    DdaJump r;
    const float guess = ((d.dd1 - d.dd0) + fmaf(kf, c.s1, c.s0)) * c.inv - 0.5f;
    float n = fminf(fmaxf((guess + 8388608.0f) - 8388608.0f, 0.0f), kf);
    float m = kf - n;
    float a0 = fmaf(n, c.s0, d.dd0), a1 = fmaf(m, c.s1, d.dd1);
    // the sums before, from the chain's start: a0 or a1 of a count too many may
    // lie past its binade, rounded to the coarser ulp, and so would a0 - s0
    const bool over = n > 0.0f && !(fmaf(n - 1.0f, c.s0, d.dd0) <= a1);
    const bool under = m > 0.0f && !(fmaf(m - 1.0f, c.s1, d.dd1) < a0);
    n += over ? -1.0f : (under ? 1.0f : 0.0f);
    m = kf - n;
    a0 = fmaf(n, c.s0, d.dd0);
    a1 = fmaf(m, c.s1, d.dd1);
    r.axis1 = a1 < a0;
    r.dd = r.axis1 ? a1 : a0;
    r.px = fmaf(r.axis1 ? m : n, r.axis1 ? c.r1 : d.g0x, r.axis1 ? d.i1x : d.i0x);
    r.py = fmaf(r.axis1 ? m : n, r.axis1 ? d.g1y : c.r0, r.axis1 ? d.i1y : d.i0y);
    n = r.axis1 ? n : n + 1.0f;
    m = (kf + 1.0f) - n;
    r.dd0 = fmaf(n, c.s0, d.dd0);
    r.i0x = fmaf(n, d.g0x, d.i0x);
    r.i0y = fmaf(n, c.r0, d.i0y);
    r.dd1 = fmaf(m, c.s1, d.dd1);
    r.i1x = fmaf(m, c.r1, d.i1x);
    r.i1y = fmaf(m, d.g1y, d.i1y);
    const uint32_t moved = (bits_of(r.dd0) ^ bits_of(d.dd0)) | (bits_of(r.dd1) ^ bits_of(d.dd1)) |
                           (bits_of(r.i0x) ^ bits_of(d.i0x)) | (bits_of(r.i0y) ^ bits_of(d.i0y)) |
                           (bits_of(r.i1x) ^ bits_of(d.i1x)) | (bits_of(r.i1y) ^ bits_of(d.i1y));
    // what an axis that takes at most one step would do next does not matter
    r.ok = (moved & 0xff800000u) == 0u && (n < 2.0f || c.steady0) && (m < 2.0f || c.steady1);
    r.kept = (n < 1.0f || c.steady0) && (m < 1.0f || c.steady1);
    return r;
}

}  // namespace rle
