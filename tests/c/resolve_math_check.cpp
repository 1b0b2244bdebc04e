// Checks csrc/resolve_math.h: the shader's texture coordinates against the
// form that keeps only the terms that count, over random cameras' uniforms and
// pixels (and pixels that share a coordinate with the vanishing point), and
// the division by a known divisor against IEEE division.  Arguments: seed,
// frames.  Prints the mismatches of either and the coordinates compared.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "resolve_math.h"

using rle::bits_of;

static int texel(float t, int size) {  // as the kernel: floor, saturating, NaN to 0
    const float v = t * static_cast<float>(size);
    if (!(v > 0)) return 0;
    return v >= static_cast<float>(size) ? size - 1 : static_cast<int>(std::floor(v));
}

int main(int argc, char** argv) {
    std::mt19937 rng(static_cast<unsigned>(argc > 1 ? std::atoi(argv[1]) : 1));
    const int frames = argc > 2 ? std::atoi(argv[2]) : 100;
    auto uni = [&](double lo, double hi) { return std::uniform_real_distribution<double>(lo, hi)(rng); };
    auto pick = [&](int n) { return static_cast<int>(rng() % static_cast<unsigned>(n)); };
    long bad = 0, bad_div = 0, seen = 0;
    for (int f = 0; f < frames; f++) {
        const int w = 8 + pick(pick(2) ? 120 : 4000), h = 8 + pick(w - 7);
        rle::ResolveGeometry g{};
        g.resx = static_cast<float>(w);
        g.resy = static_cast<float>(h);
        const double far = std::pow(10.0, uni(-1, 7));
        g.vanish_x = static_cast<float>(uni(0, 1) < 0.5 ? uni(-0.2, 1.2) : uni(-far, far));
        g.vanish_y = static_cast<float>(uni(0, 1) < 0.5 ? uni(-0.2, 1.2) : uni(-far, far));
        // on a pixel's centre, or on 0 and 1
        if (pick(4) == 0) g.vanish_x = (static_cast<float>(pick(w)) + 0.5f) / g.resx;
        if (pick(4) == 0) g.vanish_y = (static_cast<float>(pick(h)) + 0.5f) / g.resy;
        if (pick(16) == 0) g.vanish_x = static_cast<float>(pick(2));
        if (pick(16) == 0) g.vanish_y = static_cast<float>(pick(2));
        g.ofs_x = static_cast<float>(uni(-2, 2));
        g.ofs_y = static_cast<float>(uni(-2, 4));
        g.ofs_z = static_cast<float>(uni(-2, 6));
        g.ofs_w = static_cast<float>(uni(-2, 8));
        g.ratio = pick(2) ? 1.0f : static_cast<float>(uni(0.5, 2));
        g.rxg0 = static_cast<float>(pick(2));
        rle::resolve_derive(&g);
        if (!g.plain) continue;
        const int S = 8 + pick(5000), rows = 8 + pick(20000);
        for (int i = 0; i < 20000; i++) {
            const float fx = static_cast<float>(pick(w)) + 0.5f, fy = static_cast<float>(pick(h)) + 0.5f;
            float ax, ay, bx, by;
            rle::resolve_coords_shader(g, fx, fy, &ax, &ay);
            rle::resolve_coords(g, fx, fy, &bx, &by);
            if (texel(ax, S) != texel(bx, S) || texel(ay, rows) != texel(by, rows) || (ax == ax && ax != bx) ||
                (ay == ay && ay != by))
                bad++;
            seen++;
        }
        for (int i = 0; i < 20000; i++) {
            const float a = static_cast<float>(std::ldexp(uni(1, 2), pick(120) - 60));
            if (bits_of(rle::div_known(a, g.resx, g.inv_resx)) != bits_of(a / g.resx)) bad_div++;
        }
    }
    std::printf("%ld %ld %ld\n", bad, bad_div, seen);
    return 0;
}
