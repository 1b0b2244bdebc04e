// Ray buffer -> screen resolve on sm_103a.
//
// The reference warps its ray buffer onto the screen in a GLSL fragment
// shader (bin/shader/colorize_buddha_soft.frag:12-80): per pixel it finds
// the fan (up/down/left/right of the vanishing point) the pixel lies in, the
// column ray through it and the sample along that ray, then fetches the
// texel with GL_NEAREST / GL_CLAMP_TO_EDGE (src/GL_Main.cpp:152-157).  This
// kernel does the same arithmetic, one thread per pixel, as IEEE single
// operations in the shader's order (resolve_math.h; compiled with
// -fmad=false), and decodes the sample: sky, no data, or an RGB565 colour with
// its float depth.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#include "rle_internal.h"

namespace rle {
namespace {

#ifdef RLE_BOUNDS_CHECK
__device__ unsigned int g_bounds[4];
__device__ __forceinline__ bool in_bounds(bool ok, unsigned code, unsigned long long idx) {
    if (!ok) {
        const unsigned prev = atomicOr(&g_bounds[0], code);
        if (prev == 0) {
            g_bounds[1] = static_cast<unsigned>(idx);
            g_bounds[2] = static_cast<unsigned>(idx >> 32);
        }
    }
    return ok;
}
#else
__device__ __forceinline__ bool in_bounds(bool, unsigned, unsigned long long) { return true; }
#endif

// min(max((int)floor(t * size), 0), size - 1); NaN gives 0
__device__ __forceinline__ int texel(float t, int size) {
    return min(max(__float2int_rd(t * static_cast<float>(size)), 0), size - 1);
}

__device__ __forceinline__ uint32_t rgb565_to_rgba8(uint32_t c) {
    uint32_t r = (c >> 11) & 31u, g = (c >> 5) & 63u, b = c & 31u;
    r = (r << 3) | (r >> 2);
    g = (g << 2) | (g >> 4);
    b = (b << 3) | (b >> 2);
    return r | (g << 8) | (b << 16) | 0xff000000u;
}

template <bool kHits>
__device__ __forceinline__ void resolve_pixel(const ResolveParams& P, int col, int row) {
    const float fx = static_cast<float>(col) + 0.5f;
    const float fy = static_cast<float>(P.height - 1 - row) + 0.5f;  // GL rows count from the bottom
    float tx, ty;
    if (P.geo.plain) resolve_coords(P.geo, fx, fy, &tx, &ty);
    else resolve_coords_shader(P.geo, fx, fy, &tx, &ty);
    const int s = texel(tx, P.S);
    const int rr = texel(ty, P.rows);
    const size_t si = static_cast<size_t>(rr) * P.S + s;
    const size_t pi = static_cast<size_t>(row) * P.width + col;
    // rows past the rays cast hold no data (the reference's pixel buffer
    // keeps whatever an earlier frame left there)
    const bool cast = rr < P.rays && in_bounds(si < static_cast<size_t>(P.rows) * P.S, kBoundsResolve, si);
    const uint32_t w = cast ? __ldg(&P.raybuf[si]) : 0u;
    const float d = cast ? __ldg(&P.raydepth[si]) : 0.0f;
    uint32_t c;
    float dep;
    if (((w >> 16) & 0xffu) == 0xffu) {  // sky: the shader's c.z == 1.0
        c = 0xffffccb2u;
        dep = INFINITY;
    } else if (d == 0.0f) {  // outside the ray's clip range
        c = 0u;
        dep = 0.0f;
    } else {
        c = rgb565_to_rgba8(w & 0xffffu);
        dep = d;
    }
    P.colour[pi] = c;
    P.depth[pi] = dep;
    if (kHits) {
        rle_hit h = {0, 0, 0, 0, 0};
        if (P.rayhit && cast) h = P.rayhit[si];
        P.hit[pi] = h;
    }
}

// Bound by its instructions (issue slots 81% taken at 3840x2160, 74% at
// 1920x1080), with the L1 close behind (66% and 63%).  In the up and down fans
// the pixels of a screen row lie on as many column rays, a line each, and those
// of a screen column are neighbours on one ray; to the sides it is the other way
// round.  A warp takes 8x4 pixels, 4 to 8 lines per gather in either (a row of
// 32: up to 32, and the gathers bound it).  3840x2160 frames: 69 us with the
// shader's arithmetic as it stands and rows of 128, 63 us with the terms that
// count (resolve_math.h) and rows of 32, 46 us with 8x4 pixels per warp (4x8: 46,
// 16x2: 47); 1920x1080: 20, 18, 13 us.
constexpr int kTileX = 32, kTileY = 8;  // pixels of a block
constexpr int kWarpX = 8, kWarpY = 4;   // pixels of a warp
static_assert(kWarpX * kWarpY == 32 && kTileX % kWarpX == 0 && kTileY % kWarpY == 0, "tile");

// Pixel of a block's thread within its tile.
__device__ __forceinline__ int tile_col(int t) { return t / 32 % (kTileX / kWarpX) * kWarpX + t % kWarpX; }
__device__ __forceinline__ int tile_row(int t) {
    return t / 32 / (kTileX / kWarpX) * kWarpY + t % 32 / kWarpX;
}

template <bool kHits>
__global__ void __launch_bounds__(kTileX * kTileY) resolve_kernel(const __grid_constant__ ResolveParams P) {
    const int col = blockIdx.x * kTileX + tile_col(threadIdx.x);
    const int row = blockIdx.y * kTileY + tile_row(threadIdx.x);
    if (col >= P.width || row >= P.height) return;
    resolve_pixel<kHits>(P, col, row);
}

// All frames of a batch: block b belongs to the frame f with
// block_start[f] <= b < block_start[f+1] and covers 256 of its pixels.
constexpr int kResolveBlock = 256;

// Persistent: block i takes pixel blocks i, i + gridDim.x, ... of the batch, in
// rows: its gathers bound it (L1 80% taken, issue slots 40%; 99 us for eight
// 1280x720 frames, which as single frames take about half).
__global__ void __launch_bounds__(kResolveBlock) resolve_batch_kernel(const BatchHeader* __restrict__ hdr,
                                                                      const int* __restrict__ block_start,
                                                                      const ResolveParams* __restrict__ frames) {
    const int nframes = hdr->nframes;
    const int total = block_start[nframes];
    int f = 0;
    for (int b = blockIdx.x; b < total; b += gridDim.x) {
        if (b < block_start[f] || b >= block_start[f + 1]) {
            int lo = 0, hi = nframes - 1;  // last frame with block_start <= b
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (block_start[mid] <= b) lo = mid;
                else hi = mid - 1;
            }
            f = lo;
        }
        const ResolveParams& P = frames[f];
        const long long pix = static_cast<long long>(b - block_start[f]) * kResolveBlock + threadIdx.x;
        if (pix >= static_cast<long long>(P.width) * P.height) continue;
        const int row = static_cast<int>(pix / P.width), col = static_cast<int>(pix % P.width);
        if (P.hit) resolve_pixel<true>(P, col, row);
        else resolve_pixel<false>(P, col, row);
    }
}

}  // namespace

int resolve_batch_blocks(int width, int height) {
    return static_cast<int>((static_cast<long long>(width) * height + kResolveBlock - 1) / kResolveBlock);
}

bool bounds_resolve(unsigned* out4, bool clear) {
#ifdef RLE_BOUNDS_CHECK
    if (cudaMemcpyFromSymbol(out4, g_bounds, sizeof(unsigned) * 4) != cudaSuccess) return false;
    if (clear) {
        const unsigned z[4] = {0, 0, 0, 0};
        if (cudaMemcpyToSymbol(g_bounds, z, sizeof(z)) != cudaSuccess) return false;
    }
    return true;
#else
    (void)out4;
    (void)clear;
    return false;
#endif
}

rle_status launch_resolve_batch(const BatchResolve& b, void* stream) {
    if (b.blocks <= 0) return RLE_OK;
    forget_last_error();
    resolve_batch_kernel<<<b.blocks, kResolveBlock, 0, static_cast<cudaStream_t>(stream)>>>(b.header, b.block_start,
                                                                                            b.frames);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("batch resolve launch: %s", cudaGetErrorString(e));
        return RLE_ERR_CUDA;
    }
    return RLE_OK;
}

rle_status launch_resolve(const ResolveParams& p, void* stream) {
    const dim3 block(kTileX * kTileY, 1, 1);
    const dim3 grid((p.width + kTileX - 1) / kTileX, (p.height + kTileY - 1) / kTileY, 1);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    forget_last_error();
    if (p.hit) resolve_kernel<true><<<grid, block, 0, s>>>(p);
    else resolve_kernel<false><<<grid, block, 0, s>>>(p);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("resolve launch: %s", cudaGetErrorString(e));
        return RLE_ERR_CUDA;
    }
    return RLE_OK;
}

}  // namespace rle
