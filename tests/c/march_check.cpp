// Checks that calls whose rays would march for ever are refused before anything
// is launched: rle::march_ends (csrc/frame.cpp) against the march's loop on z,
// step by step, and rle_render_rays on a launcher that counts.  Arguments: seed,
// cases.  Prints the schedules judged wrongly, those that end and that do not,
// and what rle_render_rays did for a first switch distance of 0 and of 1.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "rle_internal.h"

static int launches = 0;
namespace rle {
rle_status launch_raycast(const RayParams&, void*) {
    launches++;
    return RLE_OK;
}
rle_status launch_resolve(const ResolveParams&, void*) { return RLE_OK; }
bool bounds_render(unsigned*, bool) { return false; }
bool bounds_resolve(unsigned*, bool) { return false; }
}  // namespace rle
extern "C" cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
extern "C" cudaError_t cudaSetDevice(int) { return cudaSuccess; }
extern "C" cudaError_t cudaGetLastError() { return cudaSuccess; }
extern "C" cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
extern "C" const char* cudaGetErrorString(cudaError_t) { return "fake"; }

// 1: ends, 0: does not, -1: too long to tell.  The kernel's loop (src/Cuda_Render.h:343-372).
static int march(int mapswitch, float posy, int z_far) {
    uint32_t sw = static_cast<uint32_t>(mapswitch);
    float z = 0, dz = 1, y = posy;
    for (long step = 0; step < 3000000; step++) {
        int doublings = 0;
        while (z > static_cast<float>(static_cast<int32_t>(sw)) || y > 512.0f) {
            if (++doublings > 100) return 0;
            y *= 0.5f;
            sw *= 2;
            dz *= 2;
        }
        const float before = z;
        z += dz;
        if (z > static_cast<float>(z_far)) return 1;
        if (z == before) return 0;
    }
    return -1;
}

int main(int argc, char** argv) {
    std::mt19937 rng(static_cast<unsigned>(argc > 1 ? std::atoi(argv[1]) : 1));
    const int cases = argc > 2 ? std::atoi(argv[2]) : 1000;
    auto pick = [&](int n) { return static_cast<int>(rng() % static_cast<unsigned>(n)); };
    long bad = 0, ends = 0, endless = 0;
    for (int c = 0; c < cases; c++) {
        // distances around 0, powers of two and the last whole number of a float
        int sw = pick(3) ? pick(5000) - 40 : (1 << pick(31)) + pick(3) - 1;
        if (pick(8) == 0) sw = -sw;
        const float posy = static_cast<float>(pick(2) ? pick(600) - 300 : pick(1000000));
        int z_far = pick(2) ? 1 + pick(100000) : (1 << pick(31)) + pick(3) - 1;
        if (pick(8) == 0) z_far = (1 << 24) + pick(100);
        const int want = march(sw, posy, z_far);
        if (want < 0) continue;
        (want ? ends : endless)++;
        bad += rle::march_ends(sw, posy, z_far) != (want == 1);
    }
    int status[2], launched[2];
    for (int i = 0; i < 2; i++) {
        rle_scene s;
        s.nummaps = 1;
        s.lv[0].sx = s.lv[0].sz = 8;
        rle_camera cam = {{4.5f, -40.0f, 4.5f}, {0.5f, 0.3f, 0.0f}, 90.0f};  // looks down
        rle_view_params view = {64, 64, 0, 0, 0.0f, 1 + i, 0};                // 1 * 0.25 * (4 - 0.5) is 0 as an int, 2 * ... 1
        rle_raymap rm;
        uint32_t words = 0;
        float depth = 0;
        if (rle_raymap_build(&cam, &view, &rm) != RLE_OK) return 2;
        launches = 0;
        status[i] = rle_render_rays(&s, &rm, &words, &depth, nullptr, nullptr, nullptr);
        launched[i] = launches;
    }
    std::printf("%ld %ld %ld %d %d %d %d\n", bad, ends, endless, status[0], launched[0], status[1], launched[1]);
    return 0;
}
