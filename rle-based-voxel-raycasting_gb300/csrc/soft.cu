// Soft post-filter on sm_103a: the reference's second display pass
// (bin/shader/soft.frag, drawn by src/main.cpp:627-653 over the frame
// buffer object the colorize pass filled).
//
// The colorize pass leaves, per pixel, an RGBA8 texel whose alpha is
// 0.001/z clamped to [0, 1] (z = the ray sample's depth16 as the shader reads
// it: low byte/255/256 + high byte/255; sky has alpha 0,
// colorize_buddha_soft.frag:86-136).  The soft pass then, per pixel:
//   1. takes the largest alpha among the pixel and 7 bilinear samples on a
//      circle of radius 0.005 (texture units of the 2048^2 frame buffer);
//   2. if 0.0023 * that maximum exceeds 0.00008, averages the pixel with the
//      samples of a 5x5 grid of radius 0.0023 * max whose alpha is at least
//      0.7 * max, provided more than 6 contribute; otherwise keeps the pixel.
// The frame buffer texture is RGBA8 with GL_LINEAR filtering and clamp to
// edge (src/GL_Main.h:150-165); here the bilinear weights are computed in
// single precision (a GPU's texture unit quantizes them to 8 bits, which no
// restatement reproduces) and the clamp is to the frame, not the 2048^2
// buffer.  Circle offsets and grid steps are the shader's float loops,
// evaluated once on the host.
//
// Tiling: a block filters a 32x16 tile; the texels of the tile and its apron
// (12 texels: circle radius 10.24 plus the bilinear neighbour) are built
// once into shared memory, already divided by 255 and clamped to the frame,
// then every tap reads shared memory.
//
// Bound by shared-memory reads and instructions alike (33 bilinear taps per
// pixel, 1.7 KB of shared memory where it is filtered): on a 1920x1080 frame the
// L1's data pipe is 68% and the issue slots are 69% taken, at half of the warps'
// slots.
// Unpacking RGBA8 at each tap cost 16 IEEE divisions by 255 (the kernel took
// 332 and 503 us on two 1920x1080 frames); four floats per texel cost one
// 16-byte read, and the alpha alone, which the circle needs, has a plane of its
// own (114 and 170 us).  The tap grid is a product: its 5 columns and 5 rows are
// placed once per pixel, and the channels are blended two to an instruction (85
// and 118 us, at four blocks a multiprocessor).
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#include "rle_internal.h"

namespace rle {
namespace {

constexpr int kTileX = 32, kTileY = 16, kApron = 12;
constexpr int kThreadsY = 8;  // a thread filters rows y and y + 8 of its tile
constexpr int kSmemX = kTileX + 2 * kApron, kSmemY = kTileY + 2 * kApron;
// the shader's loops: circle angles 0, step 3.1415*1.9/6 while below 2*3.1415;
// grid -1 + k*(2/5) while below 1
constexpr int kCircle = 7, kGrid = 5;

struct SoftParams {
    int width, height;
    float circle[kCircle][2];
    float grid[kGrid];
    float one;  // 1
};

__device__ __forceinline__ float over_255(uint32_t v) {
    return div_known(static_cast<float>(v), 255.0f, 1.0f / 255.0f);
}

// Frame-buffer texel of pixel (x, row-from-top) as the colorize pass leaves
// it: its RGBA8 as the texture unit reads it, n / 255 each.
__device__ __forceinline__ float4 fbo_texel(const uint32_t* colour, const float* depth, int width, int x, int row) {
    const size_t i = static_cast<size_t>(row) * width + x;
    const uint32_t c = colour[i];
    const float d = depth[i];
    uint32_t w8;
    if (isinf(d)) {
        w8 = 0;  // sky: the colorize pass leaves fragz = 0
    } else {
        const uint32_t d16 = static_cast<uint32_t>(static_cast<int>(d) & 0xfffe);
        const float z = over_255(d16 & 255u) * (1.0f / 256.0f) + over_255(d16 >> 8);
        const float fragz = 0.001f / z;
        const float f = fminf(fmaxf(fragz, 0.0f), 1.0f);
        w8 = static_cast<uint32_t>(static_cast<int>(f * 255.0f + 0.5f));
    }
    return make_float4(over_255(c & 255u), over_255((c >> 8) & 255u), over_255((c >> 16) & 255u), over_255(w8));
}

// A GL_LINEAR sample along one axis: texture coordinate t of the 2048^2 buffer
// to the first of the two texels (index in the tile, whose origin is texel
// t0; the tile repeats the frame's edge texels beyond it) and their weights.
struct Axis {
    int i;
    float w0, w1;
};
__device__ __forceinline__ Axis place(float t, int t0) {
    const float tt = t * 2048.0f - 0.5f;
    const float f = floorf(tt);
    Axis a;
    a.i = static_cast<int>(f) - t0;
    a.w1 = tt - f;
    a.w0 = 1.0f - a.w1;
    return a;
}

__device__ __forceinline__ float blend(float w00, float t00, float w10, float t10, float w01, float t01, float w11,
                                       float t11) {
    return w00 * t00 + w10 * t10 + w01 * t01 + w11 * t11;
}

// Two floats in a register pair and their IEEE single operations, two at a
// time (one instruction each).  A product followed by a sum is contracted into
// one rounding by the assembler in this form, whatever the flags say (seen in
// the results); add_product2 therefore adds the product times a 1 that only the
// launch knows.
using Pair = unsigned long long;
__device__ __forceinline__ Pair pair(float lo, float hi) {
    Pair p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(lo), "f"(hi));
    return p;
}
__device__ __forceinline__ void split(Pair p, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p));
}
__device__ __forceinline__ Pair mul2(Pair a, Pair b) {
    Pair p;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(p) : "l"(a), "l"(b));
    return p;
}
__device__ __forceinline__ Pair add2(Pair a, Pair b) {
    Pair p;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(p) : "l"(a), "l"(b));
    return p;
}
__device__ __forceinline__ Pair add_product2(Pair sum, Pair product, Pair one) {
    Pair p;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(p) : "l"(product), "l"(one), "l"(sum));
    return p;
}
__device__ __forceinline__ Pair blend2(Pair w00, Pair t00, Pair w10, Pair t10, Pair w01, Pair t01, Pair w11, Pair t11,
                                       Pair one) {
    const Pair s = add_product2(mul2(w00, t00), mul2(w10, t10), one);
    return add_product2(add_product2(s, mul2(w01, t01), one), mul2(w11, t11), one);
}

__device__ __forceinline__ uint32_t to_byte(float v) {
    const float f = fminf(fmaxf(v, 0.0f), 1.0f);
    return static_cast<uint32_t>(static_cast<int>(f * 255.0f + 0.5f));
}

__global__ void __launch_bounds__(kTileX * kThreadsY, 4) soft_kernel(const __grid_constant__ SoftParams P,
                                                                  const uint32_t* __restrict__ colour,
                                                                  const float* __restrict__ depth,
                                                                  uint32_t* __restrict__ out) {
    __shared__ ulonglong2 tile[kSmemY][kSmemX];  // red and green, blue and alpha
    __shared__ float alpha[kSmemY][kSmemX];
    // tile origin in GL texel coordinates (rows from the bottom)
    const int gx0 = blockIdx.x * kTileX - kApron, gy0 = blockIdx.y * kTileY - kApron;
    const int tid = threadIdx.y * kTileX + threadIdx.x;
    for (int i = tid; i < kSmemX * kSmemY; i += kTileX * kThreadsY) {
        const int sx = i % kSmemX, sy = i / kSmemX;
        const int x = min(max(gx0 + sx, 0), P.width - 1);
        const int y = min(max(gy0 + sy, 0), P.height - 1);
        const float4 t = fbo_texel(colour, depth, P.width, x, P.height - 1 - y);
        tile[sy][sx] = make_ulonglong2(pair(t.x, t.y), pair(t.z, t.w));
        alpha[sy][sx] = t.w;
    }
    __syncthreads();
    const int x = blockIdx.x * kTileX + threadIdx.x;
    if (x >= P.width) return;
#pragma unroll 1
    for (int ty = threadIdx.y; ty < kTileY; ty += kThreadsY) {
        const int y = blockIdx.y * kTileY + ty;
        if (y >= P.height) return;
        const float u = (static_cast<float>(x) + 0.5f) / 2048.0f, v = (static_cast<float>(y) + 0.5f) / 2048.0f;
        const ulonglong2 own = tile[y - gy0][x - gx0];
        float4 col;
        split(own.x, col.x, col.y);
        split(own.y, col.z, col.w);
        float radmax = col.w;
#pragma unroll
        for (int i = 0; i < kCircle; i++) {
            const Axis a = place(P.circle[i][0] + u, gx0), b = place(P.circle[i][1] + v, gy0);
            radmax = fmaxf(radmax, blend(a.w0 * b.w0, alpha[b.i][a.i], a.w1 * b.w0, alpha[b.i][a.i + 1], a.w0 * b.w1,
                                         alpha[b.i + 1][a.i], a.w1 * b.w1, alpha[b.i + 1][a.i + 1]));
        }
        const float rad = 0.0023f * radmax;
        if (rad > 0.00008f) {
            const Pair one = pair(P.one, P.one);
            Pair rg = own.x, ba = own.y;  // sums
            float n = 1.0f;
            const float thresh = radmax * 0.7f;
            int row[kGrid];
            Pair row0[kGrid], row1[kGrid];
#pragma unroll
            for (int ib = 0; ib < kGrid; ib++) {
                const Axis b = place(v + P.grid[ib] * rad, gy0);
                row[ib] = b.i;
                row0[ib] = pair(b.w0, b.w0);
                row1[ib] = pair(b.w1, b.w1);
            }
#pragma unroll 1
            for (int ia = 0; ia < kGrid; ia++) {
                const Axis a = place(u + P.grid[ia] * rad, gx0);
                const Pair col0 = pair(a.w0, a.w0), col1 = pair(a.w1, a.w1);
#pragma unroll
                for (int ib = 0; ib < kGrid; ib++) {
                    const ulonglong2 t00 = tile[row[ib]][a.i], t10 = tile[row[ib]][a.i + 1];
                    const ulonglong2 t01 = tile[row[ib] + 1][a.i], t11 = tile[row[ib] + 1][a.i + 1];
                    const Pair w00 = mul2(col0, row0[ib]), w10 = mul2(col1, row0[ib]);
                    const Pair w01 = mul2(col0, row1[ib]), w11 = mul2(col1, row1[ib]);
                    const Pair c_ba = blend2(w00, t00.y, w10, t10.y, w01, t01.y, w11, t11.y, one);
                    float blue, w;
                    split(c_ba, blue, w);
                    if (w >= thresh) {
                        rg = add2(rg, blend2(w00, t00.x, w10, t10.x, w01, t01.x, w11, t11.x, one));
                        ba = add2(ba, c_ba);
                        n = n + 1.0f;
                    }
                }
            }
            float4 avg;
            split(rg, avg.x, avg.y);
            split(ba, avg.z, avg.w);
            if (n > 6.0f) {
                const float inv = 1.0f / n;
                col.x = avg.x * inv;
                col.y = avg.y * inv;
                col.z = avg.z * inv;
                col.w = avg.w * inv;
            }
        }
        out[static_cast<size_t>(P.height - 1 - y) * P.width + x] =
            to_byte(col.x) | (to_byte(col.y) << 8) | (to_byte(col.z) << 16) | (to_byte(col.w) << 24);
    }
}

}  // namespace
}  // namespace rle

extern "C" rle_status rle_soft_filter(const uint32_t* d_colour, const float* d_depth, int width, int height,
                                      uint32_t* d_out, void* stream) {
    if (!d_colour || !d_depth || !d_out || width < 1 || height < 1 || width > 2048 || height > 2048 ||
        d_out == d_colour) {
        rle::set_error("rle_soft_filter: colour, depth and a separate output of 1..2048 x 1..2048 pixels required");
        return RLE_ERR_INVALID_ARG;
    }
    rle::SoftParams P;
    P.width = width;
    P.one = 1.0f;
    P.height = height;
    const float step = 3.1415f * 1.9f / 6.0f;
    float angle = 0.0f, cell = -1.0f;
    for (auto& c : P.circle) {
        c[0] = std::sin(angle) * 0.005f;
        c[1] = std::cos(angle) * 0.005f;
        angle += step;
    }
    for (float& g : P.grid) {
        g = cell;
        cell += 2.0f / 5.0f;
    }
    const dim3 block(rle::kTileX, rle::kThreadsY);
    const dim3 grid((width + rle::kTileX - 1) / rle::kTileX, (height + rle::kTileY - 1) / rle::kTileY);
    rle::forget_last_error();
    rle::soft_kernel<<<grid, block, 0, static_cast<cudaStream_t>(stream)>>>(P, d_colour, d_depth, d_out);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        rle::set_error("rle_soft_filter: %s", cudaGetErrorString(e));
        return RLE_ERR_CUDA;
    }
    return RLE_OK;
}
