// Checks csrc/cave_noise.h: the conversion-free simplex noise against
// gen::simplex3 and the cave test against gen::carved, over random points,
// lattice points and neighbours of lattice planes up to the coordinate limit.
// Arguments: seed, points.  Prints the mismatches of either and the points.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <utility>

#include "cave_noise.h"

using namespace rle::gen;

int main(int argc, char** argv) {
    std::mt19937 rng(static_cast<unsigned>(argc > 1 ? std::atoi(argv[1]) : 1));
    const long points = argc > 2 ? std::atol(argv[2]) : 1000;
    uint8_t perm[512];
    uint32_t code[512];
    for (int i = 0; i < 256; i++) perm[i] = static_cast<uint8_t>(i);
    for (int i = 255; i > 0; i--) std::swap(perm[i], perm[rng() % static_cast<unsigned>(i + 1)]);
    for (int i = 0; i < 512; i++) {
        perm[i] = perm[i & 255];
        code[i] = grad_code(perm[i]);
    }
    auto uni = [&](double hi) { return std::uniform_real_distribution<double>(0.0, hi)(rng); };
    long bad = 0, bad_cave = 0;
    for (long n = 0; n < points; n++) {
        float p[3];
        const double hi = std::exp2(uni(20.0) - 2.0);
        const unsigned how = rng() % 4;
        for (float& v : p) {
            v = static_cast<float>(uni(hi));
            if (how == 1) v = std::floor(v);                                        // lattice points
            if (how == 2) v = std::nextafterf(std::floor(v), rng() & 1 ? 2e6f : 0.0f);  // and their neighbours
            if (how == 3) v = p[0] + static_cast<float>(rng() % 3) * (rng() & 1 ? 0.5f : 0.0f);  // equal coordinates
            if (!(v > 0.0f)) v = 0.0f;
        }
        const float a = simplex3(perm, p[0], p[1], p[2]), b = cave_simplex(perm, code, p[0], p[1], p[2]);
        bad += rle::bits_of(a) != rle::bits_of(b);
        Consts c{};
        c.cave_threshold = static_cast<float>(uni(0.5));
        c.cave_period = static_cast<float>(1.0 + uni(200.0));
        const int x = static_cast<int>(uni(65535)), y = static_cast<int>(uni(1023)), z = static_cast<int>(uni(65535));
        bad_cave += carved(c, perm, x, y, z) != cave_carved(c, perm, code, 1.0f / c.cave_period, x, y, z);
    }
    std::printf("%ld %ld %ld\n", bad, bad_cave, points);
    return 0;
}
