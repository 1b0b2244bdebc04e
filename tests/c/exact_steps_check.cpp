// Checks csrc/exact_steps.h and csrc/dda.h against the plain loops they stand
// for, bit for bit, on random inputs.  Arguments: seed, cases.  Prints the
// number of mismatches of accumulate, steady_step and dda_jump, and how many
// of the latter two's cases took the closed form.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "dda.h"

using rle::bits_of;

static bool same(float a, float b) { return bits_of(a) == bits_of(b) || (a != a && b != b); }

int main(int argc, char** argv) {
    std::mt19937 rng(static_cast<unsigned>(argc > 1 ? std::atoi(argv[1]) : 1));
    const int cases = argc > 2 ? std::atoi(argv[2]) : 100000;
    auto uni = [&](double lo, double hi) { return std::uniform_real_distribution<double>(lo, hi)(rng); };
    auto pick = [&](int n) { return static_cast<int>(rng() % static_cast<unsigned>(n)); };
    long bad_acc = 0, bad_steady = 0, steady = 0, bad_dda = 0, placed = 0;
    for (int c = 0; c < cases; c++) {
        // magnitudes far apart and close, short mantissas (ties), exact powers of two, both signs
        float x = static_cast<float>(std::ldexp(uni(1, 2), pick(40) - 20)), g = static_cast<float>(std::ldexp(uni(1, 2), pick(40) - 24));
        if (pick(3) == 0) g = rle::float_of(bits_of(g) & (0xffffffffu << pick(24)));
        if (pick(3) == 0) x = rle::float_of(bits_of(x) & (0xffffffffu << pick(24)));
        if (pick(4) == 0) g = x * static_cast<float>(std::ldexp(1.0, -pick(30)));
        if (pick(2)) g = -g;
        if (pick(2)) x = -x;
        switch (pick(64)) {
            case 0: x = 0.0f; break;
            case 1: g = 0.0f; break;
            case 2: x = INFINITY; break;
            case 3: g = INFINITY; break;
            case 4: x = NAN; break;
            case 5: x = 1e-40f; break;
            case 6: g = 1e-42f; break;
            case 7: x = 3e38f; break;
        }
        const int m = pick(4) ? pick(40) : pick(3000);
        float want = x, step = 0;
        const bool ok = rle::steady_step(x, g, m, &step);
        bool all = true;
        for (int i = 1; i <= m; i++) {
            want += g;
            if (ok && !same(want, fmaf(static_cast<float>(i), step, x))) all = false;
        }
        if (!same(rle::accumulate(x, g, m), want)) bad_acc++;
        steady += ok;
        if (!all) bad_steady++;
    }
    for (int c = 0; c < cases / 50; c++) {
        double th = uni(0, 6.283185307179586);
        if (pick(3) == 0) th = pick(4) * 1.5707963267948966 + uni(-1, 1) * std::ldexp(1.0, -pick(24));
        const float dx = static_cast<float>(std::cos(th)), dy = static_cast<float>(std::sin(th));
        float px = static_cast<float>(uni(-200, 3000)), pz = static_cast<float>(uni(-200, 3000));
        if (pick(4) == 0) px = std::floor(px);
        if (pick(4) == 0) pz = std::floor(pz) + 0.5f;
        // set-up as the ray's (src/Cuda_Render.h:306-341)
        rle::Dda d{};
        float sx = -1, sy = -1, fx = px - static_cast<float>(static_cast<int>(px)), fy = pz - static_cast<float>(static_cast<int>(pz));
        if (dx >= 0) { sx = 1; fx = 1 - fx; }
        if (dy >= 0) { sy = 1; fy = 1 - fy; }
        d.g0y = dy / std::fabs(dx);
        d.g0x = sx;
        d.g1x = dx / std::fabs(dy);
        d.g1y = sy;
        d.i0x = d.g0x * fx;
        d.i0y = d.g0y * fx;
        d.i1x = d.g1x * fy;
        d.i1y = d.g1y * fy;
        d.gd0 = std::sqrt(d.g0x * d.g0x + d.g0y * d.g0y);
        d.gd1 = std::sqrt(d.g1x * d.g1x + d.g1y * d.g1y);
        d.dd0 = std::sqrt(d.i0x * d.i0x + d.i0y * d.i0y);
        d.dd1 = std::sqrt(d.i1x * d.i1x + d.i1y * d.i1y);
        rle::DdaCache cache{};
        bool cached = false;
        for (int chunk = 0; chunk < 60; chunk++) {
            const rle::Dda start = d;
            const bool can = rle::dda_can_jump(start);
            if (can && !cached) cache = rle::dda_cache(start);
            bool before_ok = can, kept = false;  // every step so far was in place
            for (int k = 0; k < 32; k++) {
                const rle::Dda at = d;
                rle::dda_step(d);
                if (!before_ok) continue;
                const rle::DdaJump j = rle::dda_jump(start, cache, static_cast<float>(k));
                if (!same(j.dd, d.dd_now) || !same(j.px, d.pnx) || !same(j.py, d.pny) ||
                    j.axis1 != (at.dd1 < at.dd0))
                    bad_dda++;
                if (j.ok && (!same(j.dd0, d.dd0) || !same(j.dd1, d.dd1) || !same(j.i0x, d.i0x) ||
                             !same(j.i0y, d.i0y) || !same(j.i1x, d.i1x) || !same(j.i1y, d.i1y)))
                    bad_dda++;
                before_ok = j.ok;
                kept = j.kept;
                placed += j.ok;
            }
            cached = before_ok && kept;  // as the kernel keeps it after a chunk in place
            if (pick(12) == 0) {  // a level switch doubles the steps
                d.g0x *= 2; d.g0y *= 2; d.g1x *= 2; d.g1y *= 2;
                d.gd0 *= 2; d.gd1 *= 2;
                cached = false;
            }
        }
    }
    std::printf("%ld %ld %ld %ld %ld\n", bad_acc, bad_steady, bad_dda, steady, placed);
    return 0;
}
