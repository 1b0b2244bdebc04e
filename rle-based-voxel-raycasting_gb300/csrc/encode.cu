// Scene building on the GPU: the seeded generator, Tree::get_mipmap's
// >= 3-of-8 rule, RLE4::compress's surface rule and run-length encoding,
// and RLE4::load's column table, as kernels over column bitsets in HBM.
//
// Working layout: one level as column bitsets, cols[(z*W + w)*sx + x] with
// W = ceil(sy/64) u64 words per column, bit j&63 of word j>>6 being voxel j
// of the column counted from the top (the reference's j,
// src/Rle4.cpp:83-88).  Equal words of neighbouring columns are neighbours, so
// a warp of columns reads and writes whole lines.  A level is encoded in four launches:
//   surface_kernel  surface bits (solid with < 27 solid in-bounds
//                   neighbours, src/Rle4.cpp:100-132) + words per column
//   scan            exclusive prefix of the words -> slab offsets (u64)
//   write_kernel    headers and colours of every column + its table entry
// All of it is integer/bit work bound by HBM traffic; the generator kernel
// (noise) is the only arithmetic-heavy part.
#include <cuda_runtime.h>

#include <cstring>
#include <vector>

#include "cave_noise.h"
#include "rle_internal.h"
#include "scenegen_math.h"

namespace {

using rle::gen::Consts;

constexpr int kThreads = 256;

rle_status cuda_fail(cudaError_t e, const char* what) {
    cudaGetLastError();  // a failed allocation must not fail the next call's launch check
    rle::set_error("%s: %s", what, cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? RLE_ERR_NO_MEMORY : RLE_ERR_CUDA;
}

inline unsigned grid_for(long long n, int threads = kThreads) {
    return static_cast<unsigned>((n + threads - 1) / threads);
}

// ---------------------------------------------------------------- level 0

struct GenArgs {
    Consts c;
    uint8_t perm[512];
    int W;
};

// One thread per column: ground fill from the fBm height, then the caves.
// Bound by the noise's instructions: two octaves at every voxel of the band.
// gen::simplex3 as it stands spends 28 conversions between integer and float
// on an octave, at an eighth of the rate of an addition; cave_simplex has none
// and no branches, and takes every grid whose coordinates fit its floor
// (kFit): 6.25 -> 3.2 ms at 2048 x 2048 x 256 with caves.  A warp covers 8 x 4
// columns, so that its lanes read few different table entries and have ground
// heights close together.
template <bool kFit>
__global__ void __launch_bounds__(kThreads) gen_columns_kernel(const __grid_constant__ GenArgs a,
                                                               uint64_t* __restrict__ cols) {
    __shared__ uint8_t perm[512];
    __shared__ uint32_t code[512];
    for (int i = threadIdx.x; i < 512; i += blockDim.x) {
        perm[i] = a.perm[i];
        if (kFit) code[i] = rle::gen::grad_code(a.perm[i]);
    }
    __syncthreads();
    const Consts& c = a.c;
    const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= static_cast<long long>(c.sx) * c.sz) return;
    // sx and sz are powers of two >= 8: whole tiles of 8 x 4
    const int lane = static_cast<int>(t & 31), tiles = c.sx >> 3;
    const long long tile = t >> 5;
    const int x = static_cast<int>(tile & (tiles - 1)) * 8 + (lane & 7);
    const int z = static_cast<int>(tile / tiles) * 4 + (lane >> 3);
    const int h = rle::gen::ground_height(c, x, z);
    int y0 = static_cast<int>(c.cave_y0), y1 = static_cast<int>(c.cave_y1);
    if (y0 < 1) y0 = 1;
    if (y1 > h) y1 = h;
    const int ground_j = c.sy - h;  // storage indices >= ground_j are solid
    const float inv = 1.0f / c.cave_period;
    uint64_t* out = cols + static_cast<long long>(z) * a.W * c.sx + x;
    for (int w = 0; w < a.W; w++) {
        const int j0 = w * 64;
        uint64_t word;
        if (ground_j <= j0) word = ~0ull;
        else if (ground_j >= j0 + 64) word = 0;
        else word = ~0ull << (ground_j - j0);
        if (c.caves && word) {
            // heights y0 <= y < y1 <-> storage j in (sy-1-y1, sy-1-y0], all solid as y1 <= h
            const int jlo = max(j0, c.sy - y1), jhi = min(j0 + 63, c.sy - 1 - y0);
            for (int j = jlo; j <= jhi; j++) {
                const int y = c.sy - 1 - j;
                const bool carve = kFit ? rle::gen::cave_carved(c, perm, code, inv, x, y, z)
                                        : rle::gen::carved(c, perm, x, y, z);
                word &= ~(static_cast<uint64_t>(carve) << (j - j0));
            }
        }
        out[static_cast<long long>(w) * c.sx] = word;
    }
}

// Reference Tree layout (bit i&7 of byte (i + j*sx + k*sx*sy) >> 3) ->
// column bitsets.  A warp covers 32 consecutive columns of one row of
// words, so each j reads 4 adjacent bytes.
__global__ void __launch_bounds__(kThreads) transpose_kernel(const uint8_t* __restrict__ bits, int sx, int sy, int sz,
                                                             int W, uint64_t* __restrict__ cols) {
    const long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const long long n = static_cast<long long>(sx) * sz * W;
    if (t >= n) return;
    const int x = static_cast<int>(t % sx);
    const long long r = t / sx;
    const int w = static_cast<int>(r % W);
    const int z = static_cast<int>(r / W);
    const long long sxy = static_cast<long long>(sx) * sy;
    uint64_t word = 0;
    const int jend = min(sy, w * 64 + 64);
    for (int j = w * 64; j < jend; j++) {
        const long long idx = x + static_cast<long long>(j) * sx + z * sxy;
        word |= static_cast<uint64_t>((bits[idx >> 3] >> (x & 7)) & 1) << (j & 63);
    }
    cols[t] = word;
}

// ----------------------------------------------------------------- mips

__device__ __forceinline__ uint32_t compact_nibble_lsbs(uint64_t v) {
    v &= 0x1111111111111111ull;
    v = (v | (v >> 3)) & 0x0303030303030303ull;
    v = (v | (v >> 6)) & 0x000F000F000F000Full;
    v = (v | (v >> 12)) & 0x000000FF000000FFull;
    v = (v | (v >> 24)) & 0x000000000000FFFFull;
    return static_cast<uint32_t>(v);
}

__device__ __forceinline__ uint32_t spread16(uint32_t v) {
    v &= 0xFFFF;
    v = (v | (v << 8)) & 0x00FF00FFu;
    v = (v | (v << 4)) & 0x0F0F0F0Fu;
    v = (v | (v << 2)) & 0x33333333u;
    v = (v | (v << 1)) & 0x55555555u;
    return v;
}

// Level m+1 from level m (Tree::get_mipmap, src/tree.h:23-85): a voxel is
// solid when >= 3 of its 8 children are.  One thread per output column;
// each input word gives 32 output bits (pairs of rows of 4 columns).
__global__ void __launch_bounds__(kThreads) halve_kernel(const uint64_t* __restrict__ a, int asx, int aW,
                                                         uint64_t* __restrict__ b, int bsx, int bsz, int bsy, int bW) {
    const long long q = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (q >= static_cast<long long>(bsx) * bsz) return;
    const int i = static_cast<int>(q % bsx), k = static_cast<int>(q / bsx);
    const uint64_t* r0 = a + static_cast<long long>(2 * k) * aW * asx + 2 * i;
    const uint64_t* r1 = r0 + static_cast<long long>(aW) * asx;
    const uint64_t m55 = 0x5555555555555555ull, m33 = 0x3333333333333333ull;
    uint64_t* dst = b + static_cast<long long>(k) * bW * bsx + i;
    uint64_t acc = 0;
    int written = 0;
    for (int w = 0; w < aW; w++) {
        const int j0 = 32 * w;
        if (j0 >= bsy) break;
        uint64_t sa = 0, sb = 0;
        // asx is even and the levels start on 256 bytes: pairs are aligned
        const ulonglong2 p0 = *reinterpret_cast<const ulonglong2*>(r0 + static_cast<long long>(w) * asx);
        const ulonglong2 p1 = *reinterpret_cast<const ulonglong2*>(r1 + static_cast<long long>(w) * asx);
        const uint64_t v4[4] = {p0.x, p0.y, p1.x, p1.y};
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const uint64_t pc = (v4[t] & m55) + ((v4[t] >> 1) & m55);  // 2-bit pair counts
            sa += pc & m33;                                          // even pairs, 4-bit fields
            sb += (pc >> 2) & m33;                                   // odd pairs
        }
        const uint64_t ga = (sa + 0x5555555555555555ull) >> 3;  // nibble >= 3 -> bit 0 of nibble
        const uint64_t gb = (sb + 0x5555555555555555ull) >> 3;
        const uint32_t bits = spread16(compact_nibble_lsbs(ga)) | (spread16(compact_nibble_lsbs(gb)) << 1);
        acc |= static_cast<uint64_t>(bits) << (j0 & 63);
        if ((j0 & 63) == 32 || w == aW - 1 || 32 * (w + 1) >= bsy) {
            written = (j0 >> 6) + 1;
            if (written == bW && (bsy & 63)) acc &= (1ull << (bsy & 63)) - 1;
            dst[static_cast<long long>(written - 1) * bsx] = acc;
            acc = 0;
        }
    }
    for (int w = written; w < bW; w++) dst[static_cast<long long>(w) * bsx] = 0;
}

// ------------------------------------------------------- surface + count

// Headers RLE4::compress emits for one finished run after `skip` empty
// voxels: 1023-skip headers, 63-solid headers, then the run's own
// (src/Rle4.cpp:166-182).
__device__ __forceinline__ int run_headers(int skip, int solid) {
    return (skip > 0 ? (skip - 1) / 1023 : 0) + (solid - 1) / 63 + 1;
}

struct LevelStats {
    unsigned long long heads, voxels, words;
    unsigned int low;  // ~j of the smallest stored j, 0 if none (all zero at the start)
};

// One thread per column, its words in order.  A voxel is interior when the
// 3x3 columns around it are solid at its height and at the two next to it:
// with A the AND of the nine columns, A & A << 1 & A >> 1.  A thread ANDs the
// three columns of its x, and takes the two next to it from the neighbouring
// lanes.  Runs are counted at the toggles of the surface bits.  Was 3 x 9
// strided loads a word and the words in local memory: 495 -> 292 us at 2048 x
// 2048 x 256, where the walk over the toggles bounds it now.
__global__ void __launch_bounds__(kThreads) surface_kernel(const uint64_t* __restrict__ cols, int sx, int sy, int sz,
                                                           int W, uint64_t* __restrict__ surf,
                                                           uint32_t* __restrict__ nwords,
                                                           uint16_t* __restrict__ nhead, LevelStats* stats) {
    const long long q = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const bool valid = q < static_cast<long long>(sx) * sz;
    const int x = static_cast<int>(q % sx), z = static_cast<int>(q / sx);
    const bool edge = x == 0 || z == 0 || x == sx - 1 || z == sz - 1;
    const bool inside = valid && z > 0 && z < sz - 1;  // has rows on both sides
    const long long row = static_cast<long long>(W) * sx;
    const uint64_t* self = cols + z * row + x;
    // AND of the columns of x (+ dx) in the three rows, word w
    auto three = [&](int w, int dx) {
        const uint64_t* n = self + static_cast<long long>(w) * sx + dx;
        return n[-row] & n[0] & n[row];
    };
    // the nine; every lane of the warp comes here
    auto nine = [&](int w) {
        uint64_t mid = 0, left, right;
        if (inside) mid = three(w, 0);
        left = __shfl_up_sync(0xffffffffu, mid, 1);
        right = __shfl_down_sync(0xffffffffu, mid, 1);
        if (inside && !edge) {
            if (lane == 0) left = three(w, -1);
            if (lane == 31) right = three(w, 1);
        }
        return mid & left & right;
    };
    unsigned long long heads = 0, voxels = 0;
    unsigned int top = 0xffffffffu;
    int nh = 0, start = 0, end = 0;
    uint64_t before = 0, open = 0;  // the word before's nine; whether its last bit was set
    uint64_t here = nine(0);
    for (int w = 0; w < W; w++) {
        const uint64_t after = w + 1 < W ? nine(w + 1) : 0;
        if (valid) {
            uint64_t v = self[static_cast<long long>(w) * sx];
            if (!edge) {
                uint64_t inner = here & ((here << 1) | (before >> 63)) & ((here >> 1) | (after << 63));
                // j = 0 and j = sy-1 have an out-of-bounds neighbour: never interior
                if (w == 0) inner &= ~1ull;
                if (w == ((sy - 1) >> 6)) inner &= ~(1ull << ((sy - 1) & 63));
                v &= ~inner;
            }
            surf[z * row + static_cast<long long>(w) * sx + x] = v;
            voxels += __popcll(v);
            for (uint64_t t = v ^ ((v << 1) | open); t; t &= t - 1) {
                const int at = w * 64 + __ffsll(static_cast<long long>(t)) - 1;
                open ^= 1;
                if (open) {
                    if (top == 0xffffffffu) top = static_cast<unsigned>(at);
                    start = at;
                } else {
                    nh += run_headers(start - end, at - start);
                    end = at;
                }
            }
            open = v >> 63;
        }
        before = here;
        here = after;
    }
    if (valid) {
        if (open) nh += run_headers(start - end, W * 64 - start);
        heads = static_cast<unsigned long long>(nh);
        nwords[q] = static_cast<uint32_t>(2 + nh + voxels);
        nhead[q] = static_cast<uint16_t>(nh);
    }
    // warp reduction, one atomic per warp
    for (int o = 16; o; o >>= 1) {
        heads += __shfl_down_sync(0xffffffffu, heads, o);
        voxels += __shfl_down_sync(0xffffffffu, voxels, o);
        top = min(top, __shfl_down_sync(0xffffffffu, top, o));
    }
    if ((threadIdx.x & 31) == 0) {
        if (heads) atomicAdd(&stats->heads, heads);
        if (voxels) atomicAdd(&stats->voxels, voxels);
        if (top != 0xffffffffu) atomicMax(&stats->low, ~top);
    }
}

// ------------------------------------------------------------------ scan

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;
constexpr int kScanChunk = kScanThreads * kScanItems;

__device__ __forceinline__ unsigned long long block_exclusive_scan(unsigned long long v,
                                                                   unsigned long long* warp_sums,
                                                                   unsigned long long* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        unsigned long long s = lane < (blockDim.x >> 5) ? warp_sums[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        warp_sums[lane] = s;  // inclusive
    }
    __syncthreads();
    const unsigned long long base = warp > 0 ? warp_sums[warp - 1] : 0;
    if (total) *total = warp_sums[(blockDim.x >> 5) - 1];
    return base + x - v;
}

// Block sums of kScanChunk-element chunks.
__global__ void __launch_bounds__(kScanThreads) scan_reduce_kernel(const uint32_t* __restrict__ v, long long n,
                                                                   unsigned long long* __restrict__ sums) {
    __shared__ unsigned long long ws[32];
    const long long base = static_cast<long long>(blockIdx.x) * kScanChunk + threadIdx.x * kScanItems;
    unsigned long long s = 0;
    for (int i = 0; i < kScanItems; i++)
        if (base + i < n) s += v[base + i];
    for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
        unsigned long long t = threadIdx.x < (blockDim.x >> 5) ? ws[threadIdx.x] : 0;
        for (int o = 16; o; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
        if (threadIdx.x == 0) sums[blockIdx.x] = t;
    }
}

// Exclusive scan of the block sums in place (one block, any count); the
// grand total goes to *total.
__global__ void __launch_bounds__(kScanThreads) scan_sums_kernel(unsigned long long* sums, long long nb,
                                                                 unsigned long long* total) {
    __shared__ unsigned long long ws[32];
    __shared__ unsigned long long chunk_total;
    unsigned long long carry = 0;
    for (long long b0 = 0; b0 < nb; b0 += kScanThreads) {
        const long long i = b0 + threadIdx.x;
        const unsigned long long v = i < nb ? sums[i] : 0;
        const unsigned long long ex = block_exclusive_scan(v, ws, &chunk_total);
        if (i < nb) sums[i] = carry + ex;
        __syncthreads();
        carry += chunk_total;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

__global__ void __launch_bounds__(kScanThreads) scan_down_kernel(const uint32_t* __restrict__ v, long long n,
                                                                 const unsigned long long* __restrict__ sums,
                                                                 unsigned long long* __restrict__ out) {
    __shared__ unsigned long long ws[32];
    const long long base = static_cast<long long>(blockIdx.x) * kScanChunk + threadIdx.x * kScanItems;
    uint32_t item[kScanItems];
    unsigned long long s = 0;
    for (int i = 0; i < kScanItems; i++) {
        item[i] = base + i < n ? v[base + i] : 0u;
        s += item[i];
    }
    unsigned long long ex = block_exclusive_scan(s, ws, nullptr) + sums[blockIdx.x];
    for (int i = 0; i < kScanItems; i++) {
        if (base + i < n) out[base + i] = ex;
        ex += item[i];
    }
}

// ----------------------------------------------------------------- write

enum ColourMode { kColourGen = 0, kColourNormal = 1, kColourVolume = 2 };

struct WriteArgs {
    Consts c;                  // generator constants (kColourGen)
    const uint64_t* cols;      // this level's solid bits (kColourNormal)
    const uint16_t* volume;    // level-0 colours, Tree layout (kColourVolume)
    int sx0, sy0;              // level-0 size (kColourVolume)
    int mode, mip;
    int sx, sy, sz, W;
    unsigned long long words;  // slab words of the level
    // ceil(2^24 / c.sy) (kColourGen): n * per_sy >> 24 is n / c.sy for n < 2^13
    // and c.sy <= 1024, as the excess, below n / 2^24, is less than 1 / c.sy;
    // with c.sy >= 64 the product stays below 2^32
    unsigned per_sy;
};

// The reference's normal-derived colour word without material bits
// (src/Rle4.cpp:134-161 with col1 == NULL): the negated centroid of the
// solid in-bounds 3x3x3 neighbours, normalised as vec3f::normalize, its y
// mapped to 0..255 and modulated by the (i ^ k) stripe pattern.
__device__ uint16_t normal_word(const WriteArgs& a, int x, int j, int z) {
    int mx = 0, my = 0, mz = 0;
    for (int dz = -1; dz <= 1; dz++) {
        const int zz = z + dz;
        if (zz < 0 || zz >= a.sz) continue;
        for (int dx = -1; dx <= 1; dx++) {
            const int xx = x + dx;
            if (xx < 0 || xx >= a.sx) continue;
            const uint64_t* n = a.cols + static_cast<long long>(zz) * a.W * a.sx + xx;
            for (int dy = -1; dy <= 1; dy++) {
                const int jj = j + dy;
                if (jj < 0 || jj >= a.sy) continue;
                if ((n[static_cast<long long>(jj >> 6) * a.sx] >> (jj & 63)) & 1) {
                    mx += dx;
                    my += dy;
                    mz += dz;
                }
            }
        }
    }
    float cx = static_cast<float>(-mx), cy = static_cast<float>(my), cz = static_cast<float>(-mz);
    const float square = cx * cx + cy * cy + cz * cz;
    if (square <= 0.00001f) {
        cy = 0.0f;
    } else {
        const float len = 1.0f / sqrtf(square);
        cy *= len;
    }
    int ny = static_cast<int>(127.0f * cy + 128.0f);
    if (ny > 255) ny = 255;
    if (ny < 0) ny = 0;
    const int scale = 1 << a.mip;
    ny = (ny * (((((x * scale) ^ (z * scale)) >> 4) & 15) + 15)) >> 5;
    if (ny > 255) ny = 255;
    if (ny < 0) ny = 0;
    return static_cast<uint16_t>(ny);
}

// Words of a warp's columns staged in shared memory at a time, and its warps
// per block (8 KB a warp).
constexpr int kStageWords = 2048;
constexpr int kWriteWarps = 4;

// One warp per 32 consecutive columns, whose words -- [run count][colour
// count][headers][colours] each -- form one contiguous range of the slab
// array.  Every lane lays out its column in the stage: counts and headers as
// they are, and for a colour the column's lane and the voxel's j.  Then the
// warp takes the stage two words a lane, works out the colours, and stores
// four bytes a lane.  The columns differ in their numbers of voxels, so that
// colouring while walking a column leaves most lanes idle; the walk is now a
// store per voxel.  (2-byte stores at the two ends of the range, which may
// share a word with the neighbouring warps'.)  A range longer than the stage
// goes in several turns, each walking the columns that reach into it.
// All levels 1290 -> 990 us at 2048 x 2048 x 256 generated, 265 -> 138 us for a
// coloured 512 x 256 x 512 volume; instructions bound it.  (Stages of 1024 and
// 1280 words, for more blocks: 2 to 4% slower in all; the voxels by set bits
// instead of by runs: 730 instead of 755 us for generated level 0, but 109
// instead of 77 us for the volume's longer runs.)
__global__ void __launch_bounds__(kWriteWarps * 32) write_kernel(const __grid_constant__ WriteArgs a,
                                                                 const uint64_t* __restrict__ surf,
                                                                 const unsigned long long* __restrict__ offsets,
                                                                 const uint32_t* __restrict__ nwords,
                                                                 const uint16_t* __restrict__ nhead,
                                                                 uint16_t* __restrict__ slabs,
                                                                 uint2* __restrict__ table) {
    constexpr uint32_t kColour = 0x80000000u;  // | lane << 16 | j
    __shared__ uint32_t stage_all[kWriteWarps][kStageWords];
    __shared__ int tints_all[kWriteWarps][32];
    uint32_t* stage = stage_all[threadIdx.x >> 5];
    int* tints = tints_all[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const long long q = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    const long long ncols = static_cast<long long>(a.sx) * a.sz;
    const bool valid = q < ncols;
    const unsigned valid_mask = __ballot_sync(0xffffffffu, valid);
    if (valid_mask == 0) return;  // a warp past the level's last column
    const int shift = __ffs(a.sx) - 1;  // sx is a power of two
    int x = 0, z = 0, nh = 0, nw = 0;
    unsigned long long ofs = 0;
    if (valid) {
        x = static_cast<int>(q) & (a.sx - 1);
        z = static_cast<int>(q >> shift);
        ofs = offsets[q];
        nw = static_cast<int>(nwords[q]);
        nh = nhead[q];
        if (a.mode == kColourGen) tints[lane] = rle::gen::tint(a.c, x << a.mip, z << a.mip);
    }
    // the warp's range: from lane 0's offset to the end of its last valid column
    const int last = 31 - __clz(valid_mask);
    const unsigned long long base = __shfl_sync(0xffffffffu, ofs, 0);
    const int from = static_cast<int>(ofs - base), to = from + nw;  // 32 columns of 2 + 1024 + 1024 words at most
    const int n = __shfl_sync(0xffffffffu, to, last);
    const long long row = static_cast<long long>(a.W) * a.sx;
    const long long q0 = q - lane;
    uint32_t first = 0;
    uint16_t* g = slabs + base;
    const int odd = static_cast<int>(base & 1);  // the slabs start on 256 bytes
    for (int w0 = 0; w0 < n; w0 += kStageWords) {
        if (valid && from < w0 + kStageWords && to > w0) {
            auto put = [&](int at, uint32_t v) {
                const unsigned i = static_cast<unsigned>(at - w0);
                if (i < static_cast<unsigned>(kStageWords)) stage[i] = v;
            };
            put(from, static_cast<uint32_t>(nh));
            put(from + 1, static_cast<uint32_t>(nw - 2 - nh));
            const uint32_t colour0 = kColour | static_cast<uint32_t>(lane << 16);
            int hp = from + 2, cp = hp + nh, start = 0, end = 0;
            auto head = [&](uint32_t h) {
                if (hp == from + 2) first = h;
                put(hp++, h);
            };
            // headers of a finished run (src/Rle4.cpp:166-182)
            auto run = [&](int r0, int r1) {
                int skip = r0 - end, solid = r1 - r0;
                for (; skip > 1023; skip -= 1023) head(1023u);
                for (; solid > 63; solid -= 63) {
                    head(63u * 1024u + static_cast<uint32_t>(skip));
                    skip = 0;
                }
                head(static_cast<uint32_t>(solid) * 1024u + static_cast<uint32_t>(skip));
                // the run's voxels, top down
                for (int j = r0; j < r1; j++) put(cp++, colour0 + static_cast<uint32_t>(j));
                end = r1;
            };
            const uint64_t* s = surf + z * row + x;
            uint64_t open = 0;
            for (int w = 0; w < a.W; w++) {
                const uint64_t v = s[static_cast<long long>(w) * a.sx];
                for (uint64_t t = v ^ ((v << 1) | open); t; t &= t - 1) {
                    const int at = w * 64 + __ffsll(static_cast<long long>(t)) - 1;
                    open ^= 1;
                    if (open) start = at;
                    else run(start, at);
                }
                open = v >> 63;
            }
            if (open) run(start, a.W * 64);
        }
        __syncwarp();
        const int m = min(n - w0, kStageWords);
        auto word = [&](int i) {
            const uint32_t v = stage[i];
            if (!(v & kColour)) return v;
            const int l = static_cast<int>(v >> 16) & 31, j = static_cast<int>(v & 0xffffu);
            const long long qc = q0 + l;
            const int cx = static_cast<int>(qc) & (a.sx - 1), cz = static_cast<int>(qc >> shift);
            if (a.mode == kColourGen) {
                const int y = a.c.sy - 1 - (j << a.mip);
                const int band = static_cast<int>(static_cast<unsigned>(y * 8) * a.per_sy >> 24);
                return static_cast<uint32_t>(
                    rle::gen::colour_in_band(a.c, tints[l], band, cx << a.mip, y, cz << a.mip));
            }
            if (a.mode == kColourNormal) return static_cast<uint32_t>(normal_word(a, cx, j, cz));
            return static_cast<uint32_t>(a.volume[(static_cast<long long>(cx) << a.mip) +
                                                  (static_cast<long long>(j) << a.mip) * a.sx0 +
                                                  (static_cast<long long>(cz) << a.mip) * a.sx0 * a.sy0]);
        };
        // kStageWords is even: the parity of the first word is that of the range
        if (odd && lane == 0) g[w0] = static_cast<uint16_t>(word(0));
        for (int i = odd + 2 * lane; i < m; i += 64) {
            const uint32_t lo = word(i);
            if (i + 1 < m) *reinterpret_cast<uint32_t*>(g + w0 + i) = lo | (word(i + 1) << 16);
            else g[w0 + i] = static_cast<uint16_t>(lo);
        }
        __syncwarp();
    }
    if (!valid) return;
    // RLE4::load's table entry (src/Rle4.cpp:285-314): the word after the
    // two counts is read as the first header even for an empty column, where
    // it is the next column's run count (or nothing past the level's end).
    if (nh == 0) first = (ofs + 2 < a.words && q + 1 < ncols) ? nhead[q + 1] : 0u;
    table[q] = make_uint2(static_cast<uint32_t>(ofs), static_cast<uint32_t>(nh) + (first << 16));
}

// ---------------------------------------------------------------- driver

struct DevLevel {
    int sx = 0, sy = 0, sz = 0, W = 0;
    uint64_t* cols = nullptr;
};

// Working buffers of the levels encoded together.
struct Scratch {
    uint64_t* surf[RLE_MAX_MIPS] = {};
    uint32_t* nwords[RLE_MAX_MIPS] = {};
    uint16_t* nhead[RLE_MAX_MIPS] = {};
    unsigned long long* offsets[RLE_MAX_MIPS] = {};
    unsigned long long* sums = nullptr;
    LevelStats* stats = nullptr;  // device, one per level
};

struct Build {
    int device = 0;
    cudaStream_t stream = nullptr;
    std::vector<DevLevel> lv;
    Scratch sc;
    int group = 0;          // levels encoded together
    void* block = nullptr;  // the levels, the scratch of one and the totals
    void* extra = nullptr;  // the scratch of the others, where they are encoded together
    ~Build() {
        if (extra) cudaFree(extra);
        if (block) cudaFree(block);
        if (stream) cudaStreamDestroy(stream);
    }
};

rle_status launch_check(const char* what) {
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? RLE_OK : cuda_fail(e, what);
}

struct Carve {
    char* at;  // null: counts only
    size_t used = 0;
    template <class T>
    void take(T*& p, size_t n) {
        p = at ? reinterpret_cast<T*>(at + used) : nullptr;
        used += (n * sizeof(T) + 255) & ~static_cast<size_t>(255);
    }
};

// Scratch of level m in slot m; slot 0 also serves the levels that are
// encoded one by one, none larger than level 0.
void lay_out_slot(Build& B, int m, Carve& c) {
    const DevLevel& L = B.lv[m];
    const size_t n = static_cast<size_t>(L.sx) * L.sz;
    c.take(B.sc.surf[m], n * L.W);
    c.take(B.sc.nwords[m], n);
    c.take(B.sc.nhead[m], n);
    c.take(B.sc.offsets[m], n);
}

void lay_out_block(Build& B, Carve& c) {
    for (DevLevel& L : B.lv) c.take(L.cols, static_cast<size_t>(L.sx) * L.sz * L.W);
    lay_out_slot(B, 0, c);
    c.take(B.sc.sums, (static_cast<size_t>(B.lv[0].sx) * B.lv[0].sz + kScanChunk - 1) / kScanChunk);
    c.take(B.sc.stats, RLE_MAX_MIPS);
}

void lay_out_extra(Build& B, Carve& c) {
    for (size_t m = 1; m < B.lv.size(); m++) lay_out_slot(B, static_cast<int>(m), c);
}

// Two allocations for the build.  The levels are encoded together, so that the
// host waits for their sizes once; where the scratch of all of them does not
// fit the device, one by one with the scratch of the largest.
rle_status alloc_levels(Build& B, int sx, int sy, int sz, int nummaps) {
    B.lv.resize(nummaps);
    for (int m = 0; m < nummaps; m++) {
        DevLevel& L = B.lv[m];
        L.sx = sx >> m;
        L.sz = sz >> m;
        L.sy = m == 0 ? sy : B.lv[m - 1].sy / 2;
        L.W = (L.sy + 63) / 64;
    }
    Carve count{nullptr};
    lay_out_block(B, count);
    const cudaError_t e = cudaMalloc(&B.block, count.used);
    if (e != cudaSuccess) {
        B.block = nullptr;
        return cuda_fail(e, "scene build: cudaMalloc(working buffers)");
    }
    Carve block{static_cast<char*>(B.block)};
    lay_out_block(B, block);
    B.group = 1;
    if (nummaps == 1) return RLE_OK;
    Carve more{nullptr};
    lay_out_extra(B, more);
    if (cudaMalloc(&B.extra, more.used) != cudaSuccess) {
        cudaGetLastError();
        B.extra = nullptr;
        return RLE_OK;
    }
    Carve extra{static_cast<char*>(B.extra)};
    lay_out_extra(B, extra);
    B.group = nummaps;
    return RLE_OK;
}

rle_status build_mips(Build& B) {
    for (size_t m = 1; m < B.lv.size(); m++) {
        const DevLevel& A = B.lv[m - 1];
        const DevLevel& L = B.lv[m];
        halve_kernel<<<grid_for(static_cast<long long>(L.sx) * L.sz), kThreads, 0, B.stream>>>(
            A.cols, A.sx, A.W, L.cols, L.sx, L.sz, L.sy, L.W);
        const rle_status st = launch_check("halve_kernel");
        if (st != RLE_OK) return st;
    }
    return RLE_OK;
}

// Surface, counts and offsets of level m into scratch slot i.
rle_status count_level(Build& B, int m, int i) {
    const DevLevel& L = B.lv[m];
    const long long n = static_cast<long long>(L.sx) * L.sz;
    const long long nb = (n + kScanChunk - 1) / kScanChunk;
    Scratch& sc = B.sc;
    rle_status st;
    surface_kernel<<<grid_for(n), kThreads, 0, B.stream>>>(L.cols, L.sx, L.sy, L.sz, L.W, sc.surf[i], sc.nwords[i],
                                                            sc.nhead[i], sc.stats + m);
    if ((st = launch_check("surface_kernel")) != RLE_OK) return st;
    scan_reduce_kernel<<<static_cast<unsigned>(nb), kScanThreads, 0, B.stream>>>(sc.nwords[i], n, sc.sums);
    if ((st = launch_check("scan_reduce_kernel")) != RLE_OK) return st;
    scan_sums_kernel<<<1, kScanThreads, 0, B.stream>>>(sc.sums, nb, &sc.stats[m].words);
    if ((st = launch_check("scan_sums_kernel")) != RLE_OK) return st;
    scan_down_kernel<<<static_cast<unsigned>(nb), kScanThreads, 0, B.stream>>>(sc.nwords[i], n, sc.sums,
                                                                                sc.offsets[i]);
    return launch_check("scan_down_kernel");
}

// Words of level m (counted in slot i) into the scene's level.
rle_status write_level(Build& B, const WriteArgs& base, rle::Level& D, int m, int i) {
    const DevLevel& L = B.lv[m];
    // zero padding after the words (the writer covers every word)
    const cudaError_t e =
        cudaMemsetAsync(reinterpret_cast<char*>(D.d_slabs) + D.words * 2, 0, rle::kSlabPadBytes, B.stream);
    if (e != cudaSuccess) return cuda_fail(e, "scene build: cudaMemsetAsync(padding)");
    WriteArgs a = base;
    a.cols = L.cols;
    a.mip = m;
    a.sx = L.sx;
    a.sy = L.sy;
    a.sz = L.sz;
    a.W = L.W;
    a.words = D.words;
    constexpr int threads = kWriteWarps * 32;
    write_kernel<<<grid_for(static_cast<long long>(L.sx) * L.sz, threads), threads, 0, B.stream>>>(
        a, B.sc.surf[i], B.sc.offsets[i], B.sc.nwords[i], B.sc.nhead[i], D.d_slabs,
        reinterpret_cast<uint2*>(D.d_table));
    return launch_check("write_kernel");
}

// Encodes every level into the scene, B.group levels at a time.
rle_status encode_into(Build& B, const WriteArgs& base, rle_scene* s) {
    const int nummaps = static_cast<int>(B.lv.size());
    cudaError_t e = cudaMemsetAsync(B.sc.stats, 0, sizeof(LevelStats) * RLE_MAX_MIPS, B.stream);
    if (e != cudaSuccess) return cuda_fail(e, "scene build: cudaMemsetAsync");
    long long top_all = 0x7fffffffLL;
    LevelStats stats[RLE_MAX_MIPS];
    for (int m0 = 0; m0 < nummaps; m0 += B.group) {
        const int m1 = m0 + B.group < nummaps ? m0 + B.group : nummaps;
        rle_status st;
        for (int m = m0; m < m1; m++)
            if ((st = count_level(B, m, m - m0)) != RLE_OK) return st;
        if ((e = cudaMemcpyAsync(stats, B.sc.stats, sizeof(stats), cudaMemcpyDeviceToHost, B.stream)) != cudaSuccess ||
            (e = cudaStreamSynchronize(B.stream)) != cudaSuccess)
            return cuda_fail(e, "scene build: level totals");
        for (int m = m0; m < m1; m++) {
            const LevelStats& ls = stats[m];
            if (ls.words > 0xffffffffull) {
                rle::set_error("scene build: level %d needs %llu slab words (the column table holds 32-bit offsets)",
                               m, ls.words);
                return RLE_ERR_CAPACITY;
            }
            rle::Level& D = s->lv[m];
            D.sx = B.lv[m].sx;
            D.sy = B.lv[m].sy;
            D.sz = B.lv[m].sz;
            D.words = ls.words;
            s->device_bytes += static_cast<size_t>(D.sx) * D.sz * 8 + static_cast<size_t>(D.words) * 2 +
                               rle::kSlabPadBytes;
            if (m == 0) {
                s->run_headers = ls.heads;
                s->surface_voxels = ls.voxels;
            }
            // same clamp as the loader: an empty level reports INT_MAX
            const unsigned int low = ~ls.low;
            const int top = low > 0x7fffffffu ? 0x7fffffff : static_cast<int>(low);
            const long long top0 = static_cast<long long>(top) << m;
            if (top0 < top_all) top_all = top0;
        }
        if ((e = rle::alloc_scene_levels(s, m0, m1)) != cudaSuccess) {
            if (e != cudaErrorMemoryAllocation || B.group == 1)
                return cuda_fail(e, "scene build: cudaMalloc(tables and slabs)");
            // no room beside the scratch of all levels: again, one by one
            cudaGetLastError();
            cudaFree(B.extra);
            B.extra = nullptr;
            B.group = 1;
            s->device_bytes = 0;
            return encode_into(B, base, s);
        }
        for (int m = m0; m < m1; m++)
            if ((st = write_level(B, base, s->lv[m], m, m - m0)) != RLE_OK) return st;
    }
    if ((e = cudaStreamSynchronize(B.stream)) != cudaSuccess) return cuda_fail(e, "scene build");
    s->top_index = static_cast<int>(top_all);
    return RLE_OK;
}

rle_status encode_levels(Build& B, const WriteArgs& base, rle_scene** out) {
    rle_scene* s = new (std::nothrow) rle_scene();
    if (!s) return RLE_ERR_NO_MEMORY;
    s->device = B.device;
    s->nummaps = static_cast<int>(B.lv.size());
    s->height = B.lv[0].sy;
    const rle_status st = encode_into(B, base, s);
    if (st != RLE_OK) {
        cudaStreamSynchronize(B.stream);  // launched writes end before their memory goes
        rle_scene_free(s);
        return st;
    }
    *out = s;
    return RLE_OK;
}

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard() { cudaGetDevice(&prev); }
    ~DeviceGuard() {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

rle_status begin(Build& B, int device) {
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDeviceCount");
    if (device < 0 || device >= ndev) {
        rle::set_error("scene build: device %d of %d", device, ndev);
        return RLE_ERR_INVALID_ARG;
    }
    B.device = device;
    rle::forget_last_error();
    if ((e = cudaSetDevice(device)) != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
    if ((e = cudaStreamCreateWithFlags(&B.stream, cudaStreamNonBlocking)) != cudaSuccess)
        return cuda_fail(e, "cudaStreamCreate");
    return RLE_OK;
}

// Orders the build behind what is queued on `stream` (of the build's device) so
// far.  A stream that is being captured has run nothing that could be waited for.
rle_status order_behind(Build& B, cudaStream_t stream) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    cudaError_t e = cudaStreamIsCapturing(stream, &capture);
    if (e == cudaErrorStreamCaptureImplicit || capture != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return RLE_OK;
    }
    if (e == cudaSuccess) e = cudaStreamQuery(stream);
    if (e == cudaSuccess) return RLE_OK;  // nothing queued (the usual case)
    cudaEvent_t done = nullptr;
    if (e == cudaErrorNotReady) {
        cudaGetLastError();
        e = cudaEventCreateWithFlags(&done, cudaEventDisableTiming);
    }
    if (e == cudaSuccess) e = cudaEventRecord(done, stream);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(B.stream, done, 0);
    if (done) cudaEventDestroy(done);
    return e == cudaSuccess ? RLE_OK : cuda_fail(e, "scene build: ordering behind the caller's stream");
}

}  // namespace

extern "C" rle_status rle_scenegen_device(const rle_scenegen_params* p, int device, rle_scene** out) {
    if (!out) return RLE_ERR_INVALID_ARG;
    *out = nullptr;
    rle_status st = rle::scenegen_check(p);
    if (st != RLE_OK) return st;
    DeviceGuard guard;
    Build B;
    if ((st = begin(B, device)) != RLE_OK) return st;
    if ((st = alloc_levels(B, p->sx, p->sy, p->sz, p->nummaps)) != RLE_OK) return st;
    GenArgs g;
    g.c = rle::scenegen_consts(*p);
    rle::scenegen_perm(p->seed, g.perm);
    g.W = B.lv[0].W;
    const unsigned blocks = grid_for(static_cast<long long>(p->sx) * p->sz);
    if (rle::gen::cave_coords_fit(g.c)) gen_columns_kernel<true><<<blocks, kThreads, 0, B.stream>>>(g, B.lv[0].cols);
    else gen_columns_kernel<false><<<blocks, kThreads, 0, B.stream>>>(g, B.lv[0].cols);
    if ((st = launch_check("gen_columns_kernel")) != RLE_OK) return st;
    if ((st = build_mips(B)) != RLE_OK) return st;
    WriteArgs a;
    std::memset(&a, 0, sizeof(a));
    a.c = g.c;
    a.mode = kColourGen;
    a.per_sy = ((1u << 24) + static_cast<unsigned>(p->sy) - 1u) / static_cast<unsigned>(p->sy);
    return encode_levels(B, a, out);
}

namespace {

// `ordered`: behind the work queued on `stream`.
rle_status encode_device(const uint8_t* d_bits, const uint16_t* d_colours, int sx, int sy, int sz, int nummaps,
                         int device, bool ordered, cudaStream_t stream, rle_scene** out) {
    if (!out) return RLE_ERR_INVALID_ARG;
    *out = nullptr;
    auto pow2 = [](int v) { return v >= 8 && (v & (v - 1)) == 0; };
    if (!d_bits || !pow2(sx) || !pow2(sz) || sx > 65536 || sz > 65536 || sy < 1 || sy > 1024 || nummaps < 1 ||
        nummaps > RLE_MAX_MIPS || (sx >> (nummaps - 1)) < 1 || (sz >> (nummaps - 1)) < 1 ||
        (sy >> (nummaps - 1)) < 1) {
        rle::set_error("rle_encode_device: bits required; sx, sz powers of two in 8..65536, sy in 1..1024, "
                       "1..%d levels that keep every dimension >= 1",
                       RLE_MAX_MIPS);
        return RLE_ERR_INVALID_ARG;
    }
    DeviceGuard guard;
    Build B;
    rle_status st = begin(B, device);
    if (st != RLE_OK) return st;
    if (ordered && (st = order_behind(B, stream)) != RLE_OK) return st;
    if ((st = alloc_levels(B, sx, sy, sz, nummaps)) != RLE_OK) return st;
    const long long n = static_cast<long long>(sx) * sz * B.lv[0].W;
    transpose_kernel<<<grid_for(n), kThreads, 0, B.stream>>>(d_bits, sx, sy, sz, B.lv[0].W, B.lv[0].cols);
    if ((st = launch_check("transpose_kernel")) != RLE_OK) return st;
    if ((st = build_mips(B)) != RLE_OK) return st;
    WriteArgs a;
    std::memset(&a, 0, sizeof(a));
    a.mode = d_colours ? kColourVolume : kColourNormal;
    a.volume = d_colours;
    a.sx0 = sx;
    a.sy0 = sy;
    return encode_levels(B, a, out);
}

}  // namespace

extern "C" rle_status rle_encode_device(const uint8_t* d_bits, const uint16_t* d_colours, int sx, int sy, int sz,
                                        int nummaps, int device, rle_scene** out) {
    return encode_device(d_bits, d_colours, sx, sy, sz, nummaps, device, false, nullptr, out);
}

extern "C" rle_status rle_encode_device_after(const uint8_t* d_bits, const uint16_t* d_colours, int sx, int sy, int sz,
                                              int nummaps, int device, void* stream, rle_scene** out) {
    return encode_device(d_bits, d_colours, sx, sy, sz, nummaps, device, true, static_cast<cudaStream_t>(stream), out);
}
