// Checks div_known of csrc/resolve_math.h against IEEE division: every mantissa
// of the dividend (both scale alike with powers of two) by each divisor given.
// Prints the quotients that differ and those compared.
#include <cstdio>
#include <cstdlib>

#include "resolve_math.h"

int main(int argc, char** argv) {
    long bad = 0, seen = 0;
    for (int i = 1; i < argc; i++) {
        const float b = static_cast<float>(std::atof(argv[i])), inv = 1.0f / b;
        for (uint32_t m = 0; m < (1u << 23); m++, seen++) {
            const float a = rle::float_of(0x3f800000u | m);
            bad += rle::bits_of(rle::div_known(a, b, inv)) != rle::bits_of(a / b);
        }
    }
    std::printf("%ld %ld\n", bad, seen);
    return 0;
}
