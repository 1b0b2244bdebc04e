// Checks csrc/exact_steps.h against the plain loops it stands for, bit for
// bit, on random inputs.  Arguments: seed, cases.  Prints the number of
// mismatches of accumulate and steady_step, and how many of the latter's cases
// took the closed form.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "exact_steps.h"

using rle::bits_of;

static bool same(float a, float b) { return bits_of(a) == bits_of(b) || (a != a && b != b); }

int main(int argc, char** argv) {
    std::mt19937 rng(static_cast<unsigned>(argc > 1 ? std::atoi(argv[1]) : 1));
    const int cases = argc > 2 ? std::atoi(argv[2]) : 100000;
    auto uni = [&](double lo, double hi) { return std::uniform_real_distribution<double>(lo, hi)(rng); };
    auto pick = [&](int n) { return static_cast<int>(rng() % static_cast<unsigned>(n)); };
    long bad_acc = 0, bad_steady = 0, steady = 0;
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
    std::printf("%ld %ld %ld\n", bad_acc, bad_steady, steady);
    return 0;
}
