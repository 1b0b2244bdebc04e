// Which ray-buffer sample a screen pixel shows: the texture coordinates of the
// colorize shader (bin/shader/colorize_buddha_soft.frag:12-80), in its
// single-precision operations and order.  Compiled by nvcc for the kernels and
// by the host compiler for the tests.
#pragma once

#include "exact_steps.h"

namespace rle {

// Uniforms of one frame and what follows from them alone.
struct ResolveGeometry {
    float resx, resy;
    float vanish_x, vanish_y;
    float ofs_x, ofs_y, ofs_z, ofs_w;
    float ratio;
    float rxg0;        // rotation.x > 0: 1, else 0
    // derived (resolve_derive)
    float border;                // (resx - resy) / (resx * 2)
    float inv_resx, inv_resy;    // 1 / resx, 1 / resy, rounded
    int plain;                   // resolve_coords applies
};

RLE_STEP_FN float resolve_step(float edge, float x) { return x < edge ? 0.0f : 1.0f; }

// The shader's arithmetic as it stands.
RLE_STEP_FN void resolve_coords_shader(const ResolveGeometry& g, float fx, float fy, float* tx_out, float* ty_out) {
    const float RESX = g.resx, RESY = g.resy;
    const float scx = fx / RESX, scy = fy / RESY;
    const float border = (RESX - RESY) / (RESX * 2);
    const float scx1 = scx - g.vanish_x, scy1 = scy - g.vanish_y;
    const float upper = resolve_step(scy1, 0.0f);
    const float left = resolve_step(scx1, 0.0f);
    const float ostep = resolve_step(fabsf(scy1) - fabsf(scx1) * RESX / RESY, 0.0f);
    const float seg_up = (1 - upper) * (1 - ostep);
    const float seg_dn = upper * (1 - ostep);
    const float seg_rt = (1 - left) * ostep;
    const float seg_lt = left * ostep;
    const float o2 = (ostep * fx + (1 - ostep) * fy) / RESX;
    const float ang2 = scx1 * fabsf(1 - resolve_step(scy1, 0.0f) - g.vanish_y) / scy1 +
                       resolve_step(scy1, 0.0f) * (1 - g.vanish_x) + (1 - resolve_step(scy1, 0.0f)) * g.vanish_x;
    float ang3 = scy1 * fabsf(1 - resolve_step(scx1, 0.0f) - g.vanish_x) / scx1 +
                 resolve_step(scx1, 0.0f) * (1 - g.vanish_y) + (1 - resolve_step(scx1, 0.0f)) * g.vanish_y;
    ang3 = ang3 * RESY / RESX + border;
    const float x_pre = ostep * ang3 + ang2 * (1 - ostep);
    const float ty = seg_dn * (g.ofs_y + x_pre) + seg_up * (g.ofs_x + 1.0f - x_pre) + seg_lt * (g.ofs_w + x_pre) +
                     seg_rt * (g.ofs_z + 1.0f - x_pre);
    *ty_out = ty * g.ratio * 0.25f;
    const float r = g.rxg0;
    const float seg_up_x = r * seg_up + (1.0f - r) * seg_dn;
    const float seg_dn_x = r * seg_dn + (1.0f - r) * seg_up;
    const float seg_rt_x = r * seg_rt + (1.0f - r) * seg_lt;
    const float seg_lt_x = r * seg_lt + (1.0f - r) * seg_rt;
    *tx_out = seg_up_x * (o2 + border) + seg_dn_x * (1.0f - (o2 + border)) + seg_rt_x * o2 + seg_lt_x * (1.0f - o2);
}

// a / b, correctly rounded, for a divisor whose rounded reciprocal is known:
// one product and one correction with its exact remainder (Markstein, IBM J.
// Res. Dev. 34, 1990; Brisebarre, Muller and Raina, IEEE Trans. Comput. 53,
// 2004), without the range tests of a general division.  Quotient and
// remainder have to stay clear of the subnormals.
RLE_STEP_FN float div_known(float a, float b, float inv) {
    const float q = a * inv;
    return fmaf(fmaf(-q, b, a), inv, q);
}

// The same coordinates with only the terms that count: of the four fans (up,
// down, left, right of the vanishing point) a pixel lies in one, and the
// shader's weights are 1 for it and 0 for the others.  0 times a finite term
// adds nothing; what is infinite is the other axis's quotient where the pixel
// shares a coordinate with the vanishing point, and there ty is NaN.  Where
// `plain` holds nothing else overflows or comes near the subnormals.
RLE_STEP_FN void resolve_coords(const ResolveGeometry& g, float fx, float fy, float* tx_out, float* ty_out) {
    const float scx = div_known(fx, g.resx, g.inv_resx), scy = div_known(fy, g.resy, g.inv_resy);
    const float scx1 = scx - g.vanish_x, scy1 = scy - g.vanish_y;
    // fans to the side (along x), else up or down
    const bool side = !(0.0f < fabsf(scy1) - div_known(fabsf(scx1) * g.resx, g.resy, g.inv_resy));
    const float along = side ? scy1 : scx1, across = side ? scx1 : scy1;
    const bool low = !(0.0f < across);  // left or down
    const float v = side ? g.vanish_x : g.vanish_y, w = side ? g.vanish_y : g.vanish_x;
    float ang = along * fabsf(low ? 0.0f - v : 1.0f - v) / across + (low ? 1.0f - w : w);
    if (side) ang = div_known(ang * g.resy, g.resx, g.inv_resx) + g.border;
    float ty = low ? (side ? g.ofs_w : g.ofs_y) + ang : (side ? g.ofs_z : g.ofs_x) + 1.0f - ang;
    ty = ty * g.ratio * 0.25f;
    if (scx1 == 0.0f || scy1 == 0.0f) ty = float_of(0x7fffffffu);
    const float o = side ? scx : div_known(fy, g.resx, g.inv_resx) + g.border;
    *ty_out = ty;
    *tx_out = low != (g.rxg0 != 0.0f) ? o : 1.0f - o;
}

// Fills the derived fields.  The bounds of `plain` hold for every ray map of a
// camera (screens of 8 to 16384 pixels; a vanishing point is at most about 1e8
// screens away): then |scx1| and |scy1| are 0 or at least 2^-48, and no term
// exceeds 1e32.
inline void resolve_derive(ResolveGeometry* g) {
    g->border = (g->resx - g->resy) / (g->resx * 2);
    g->inv_resx = 1.0f / g->resx;
    g->inv_resy = 1.0f / g->resy;
    auto within = [](float v, float bound) { return std::fabs(v) <= bound; };
    g->plain = g->resx >= 8 && g->resy >= 8 && g->resx <= 16384 && g->resy <= 16384 && within(g->vanish_x, 1e8f) &&
               within(g->vanish_y, 1e8f) && within(g->ofs_x, 1e8f) && within(g->ofs_y, 1e8f) &&
               within(g->ofs_z, 1e8f) && within(g->ofs_w, 1e8f) && within(g->ratio, 1e8f);
}

}  // namespace rle
