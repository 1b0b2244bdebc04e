// Checks dda_jump of csrc/dda.h against the plain steps, bit for bit, on rays
// whose two axes meet at equal distances: directions in small whole-number
// ratios (45 degrees among them) from eyes at multiples of 1/16 of a cell.
// Arguments: seed, rays.  Prints the number of events and states that differ,
// of events at the first step out of place (used by the kernel, too) that were
// compared, and of ties among those.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "dda.h"

using rle::bits_of;

static bool same(float a, float b) { return bits_of(a) == bits_of(b) || (a != a && b != b); }

int main(int argc, char** argv) {
    std::mt19937 rng(static_cast<unsigned>(argc > 1 ? std::atoi(argv[1]) : 1));
    const int rays = argc > 2 ? std::atoi(argv[2]) : 20000;
    auto pick = [&](int n) { return static_cast<int>(rng() % static_cast<unsigned>(n)); };
    long bad = 0, edges = 0, ties = 0;
    for (int c = 0; c < rays; c++) {
        // the direction as it is, or divided by its length
        float dx = static_cast<float>(1 + pick(8)), dy = pick(4) ? static_cast<float>(1 + pick(8)) : dx;
        if (pick(2)) {
            const float inv = 1.0f / std::sqrt(dx * dx + dy * dy);
            dx *= inv;
            dy *= inv;
        }
        if (pick(2)) dx = -dx;
        if (pick(2)) dy = -dy;
        const int grain = 1 << pick(5);
        const float px = static_cast<float>(pick(1024 * grain)) / static_cast<float>(grain);
        const float pz = static_cast<float>(pick(1024 * grain)) / static_cast<float>(grain);
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
        for (int jump = 0; jump < 40; jump++) {
            // a jump from here, as far as it is in place and 32 steps at most,
            // and the event at the first step that is not
            const rle::Dda start = d;
            const rle::DdaCache cache = rle::dda_cache(start);
            const int steps = pick(4) ? 32 : 1 + pick(32);
            for (int k = 0; k < steps; k++) {
                const rle::Dda at = d;
                rle::dda_step(d);
                const rle::DdaJump j = rle::dda_jump(start, cache, static_cast<float>(k));
                if (!j.ok) {
                    edges++;
                    ties += at.dd0 == at.dd1;
                }
                if (!same(j.dd, d.dd_now) || !same(j.px, d.pnx) || !same(j.py, d.pny) || j.axis1 != (at.dd1 < at.dd0))
                    bad++;
                if (!j.ok) break;
                if (!same(j.dd0, d.dd0) || !same(j.dd1, d.dd1) || !same(j.i0x, d.i0x) || !same(j.i0y, d.i0y) ||
                    !same(j.i1x, d.i1x) || !same(j.i1y, d.i1y))
                    bad++;
            }
            if (pick(16) == 0) {  // a level switch doubles the steps
                d.g0x *= 2; d.g0y *= 2; d.g1x *= 2; d.g1y *= 2;
                d.gd0 *= 2; d.gd1 *= 2;
            }
        }
    }
    std::printf("%ld %ld %ld\n", bad, edges, ties);
    return 0;
}
