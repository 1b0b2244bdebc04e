// Column-ray traversal on sm_103a.
//
// Algorithm (Render::render_line, src/Cuda_Render.h:96-737, with the
// switches FLOATING_HORIZON, XFLOATING_HORIZON and SHAREMEMCLIP of
// src/core.h:24-32): a column ray marches the 2D grid of RLE columns with a
// 2D DDA, picks the mip level by distance, walks each visited column's run
// headers, projects solid runs to screen spans and fills them with
// perspective-correct colour and depth, culling with a floating horizon and
// an occupancy bitmask.
//
// Parallel decomposition: a warp owns one ray.  The ray is processed in chunks
// of 32 DDA steps, the next chunk's DDA and table fetches issued before this
// chunk's merge:
//   1. lane k finds the state of step k of the DDA (a chain of IEEE additions
//      per axis) without taking the steps before it, derives its cell and
//      fetches the column-table entry; the state before it comes from lane
//      k-1;
//   2. each lane, in parallel, tests its cell against the horizon at the start
//      of the chunk; where one passes, it scans its column's runs and records
//      in shared memory the runs the walk could still draw;
//   3. the recorded runs, in the order of the walk, go to the lanes, each of
//      which claims the samples that its span covers first in the bitmask;
//      the claimed samples are coloured later, 32 at a time.  Only a cell
//      whose outcome could depend on the horizon at its very turn is walked
//      in sequence (scan_runs).
// The pre-cull is conservative: the horizon only closes (ymin grows, ymax
// shrinks), so a cell or run culled at the chunk start would be culled at
// its turn too.  The result is the sequential algorithm's, bit for bit.
//
// Arithmetic: compiled with -fmad=false and IEEE division/square root, each
// float operation is the single IEEE operation the reference performs, in
// its order.  Per-frame sines/cosines come precomputed from the host.
//
// Output, per ray row (ray-major, S samples): every sample is written once
// -- coloured samples when drawn, the rest in a final coalesced pass (sky
// 0x00ff8844 inside the ray's clip range, 0 outside), guided by the bitmask.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#include "dda.h"
#include "exact_steps.h"
#include "rle_internal.h"

namespace rle {
namespace {

constexpr uint32_t kSky = 0x00ff8844u;

// Debug builds with RLE_BOUNDS_CHECK range-check every column-table, slab
// and ray-buffer index: a failed check records its code (and the first
// index) in g_bounds and skips the access (reads return 0) instead of
// touching memory outside the scene or the frame.
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

struct Counts {
    unsigned long long cells = 0, fetched = 0, headers = 0, runs = 0, spans = 0, pixels = 0;
};

struct F3 {
    float x, y, z;
};
__device__ __forceinline__ F3 f3(float x, float y, float z) { return F3{x, y, z}; }
__device__ __forceinline__ F3 add(F3 a, F3 b) { return f3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ F3 sub(F3 a, F3 b) { return f3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ F3 mul(F3 a, float s) { return f3(a.x * s, a.y * s, a.z * s); }

// Render::LineScale (src/Cuda_Render.h:39-52)
__device__ __forceinline__ float line_scale(F3 in, F3 c, float cmax, float cmin) {
    float sx = 1, sy = 1;
    if (c.x > 1) sx = (1 - in.x) / (c.x - in.x);
    if (c.x < 0) sx = in.x / (in.x - c.x);
    if (c.y > cmax) sy = (cmax - in.y) / (c.y - in.y);
    if (c.y < cmin) sy = (-cmin + in.y) / (in.y - c.y);
    return (sx < sy) ? sx : sy;
}

__device__ __forceinline__ F3 to3d(const RayParams& P, F3 v) {
    return f3(P.to3d[0][0] * v.x + P.to3d[1][0] * v.y + P.to3d[2][0] * v.z + P.to3d[3][0],
              P.to3d[0][1] * v.x + P.to3d[1][1] * v.y + P.to3d[2][1] * v.z + P.to3d[3][1],
              P.to3d[0][2] * v.x + P.to3d[1][2] * v.y + P.to3d[2][2] * v.z + P.to3d[3][2]);
}

// Device-wide nanosecond clock and the SM a thread runs on (profiling).
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ uint32_t sm_id() {
    uint32_t s;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(s));
    return s;
}

// One warp owns one ray.  (Two or four rays per warp share its instructions
// only while they take the same branches; the chunk that draws, the jump that
// ends early and the ray that ends are branches.  Measured on batches, 8 / 16 /
// 32 lanes per ray: 64 mixed frames 7.85 / 6.33 / 4.58 ms, eight 4K frames 3.25 /
// 3.03 / 2.42 ms, 96 frames of 96x64 2.38 / 1.24 / 0.71 ms, persistent likewise.)
constexpr int kLanes = 32;
constexpr unsigned kWarp = 0xffffffffu;

// Occupancy bitmask of one ray in shared memory (1 bit per sample).
struct Mask {
    uint32_t* w;
    __device__ __forceinline__ bool get(int y) const { return (w[y >> 5] >> (y & 31)) & 1u; }
    // first y in [y, end) whose bit is clear, or end
    __device__ __forceinline__ int first_clear(int y, int end) const {
        while (y < end) {
            const uint32_t free_bits = ~w[y >> 5] >> (y & 31);
            if (free_bits) {
                const int r = y + (__ffs(free_bits) - 1);
                return r < end ? r : end;
            }
            y = (y | 31) + 1;
        }
        return end;
    }
    // one past the last y in [begin, end) whose bit is clear, or begin
    __device__ __forceinline__ int last_clear(int begin, int end) const {
        while (end > begin) {
            const uint32_t free_bits = ~w[(end - 1) >> 5] << (31 - ((end - 1) & 31));
            if (free_bits) {
                const int r = end - __clz(free_bits);
                return r > begin ? r : begin;
            }
            end = (end - 1) & ~31;
        }
        return begin;
    }
};

// Per-ray constants after set-up.
struct Ray {
    float ray_x, ray_z;
    float rmul;          // res_x2_mul_reverse (with the field-of-view focal length)
    float pos3d_z_add, pos3d_y_add;
    int fix_x, fix_z;
    bool vertical;
    int ymin, ymax;      // clip range at the start (ymax < ymin: the ray is empty)
};

// Ray set-up: fan, 2D line, 3D direction, sample range, DDA start
// (src/Cuda_Render.h:129-304).  Returns false if the ray covers no samples.
__device__ __forceinline__ bool setup_ray(const RayParams& P, int x, Ray& R, Dda& D) {
    const int S = P.S;
    const int r0 = P.res[0], r1 = P.res[1] + r0, r2 = P.res[2] + r1;
    int q = 0;
    if (x >= r2) q = 3;
    else if (x >= r1) q = 2;
    else if (x >= r0) q = 1;
    float qofs = static_cast<float>(x);
    if (q == 1) qofs -= static_cast<float>(r0);
    if (q == 2) qofs -= static_cast<float>(r1);
    if (q == 3) qofs -= static_cast<float>(r2);
    const float a = qofs / static_cast<float>(P.res[q]);
    F3 p1 = f3(P.p5x, P.p5y, P.p5z);
    const F3 n0 = f3(P.p_no[2 * q][0], P.p_no[2 * q][1], P.p_no[2 * q][2]);
    const F3 n1 = f3(P.p_no[2 * q + 1][0], P.p_no[2 * q + 1][1], P.p_no[2 * q + 1][2]);
    F3 p2 = add(n0, mul(sub(n1, n0), a));
    {  // ClipLine (src/Cuda_Render.h:54-65)
        float s = line_scale(p1, p2, P.clip_max, P.clip_min);
        const F3 c2 = add(p1, mul(sub(p2, p1), s));
        s = line_scale(p2, p1, P.clip_max, P.clip_min);
        const F3 c1 = add(p2, mul(sub(p1, p2), s));
        p1 = c1;
        p2 = c2;
    }
    const F3 p1_3d = to3d(P, mul(p1, 4.0f));
    const F3 p2_3d = to3d(P, mul(p2, 4.0f));
    F3 d = sub(mul(add(p1_3d, p2_3d), 0.5f), f3(P.p4[0], P.p4[1], P.p4[2]));
    d.y = 0;
    {
        const float inv = 1.0f / sqrtf(d.x * d.x + d.y * d.y + d.z * d.z);
        d = mul(d, inv);
    }
    {
        const float xx = P.cos_ny * d.x + P.sin_ny * d.z;
        const float zz = P.cos_ny * d.z - P.sin_ny * d.x;
        d.x = xx;
        d.z = zz;
    }
    R.ray_x = d.x;
    R.ray_z = d.z;
    R.vertical = q < 2;
    const float sin_x = P.sin_x, cos_x = P.cos_x;

    bool reverse = false;
    if (R.vertical && R.ray_z <= 0) reverse = true;
    if (!R.vertical && R.ray_x <= 0 && sin_x > 0) reverse = true;
    if (!R.vertical && R.ray_x > 0 && sin_x < 0) reverse = true;
    float rmul = reverse ? -P.focal : P.focal;
    if (R.vertical) rmul = -rmul;
    R.rmul = rmul;
    R.pos3d_z_add = sin_x;
    R.pos3d_y_add = (R.vertical ? cos_x : 0.0f) * rmul;
    R.ymin = 0;
    R.ymax = -1;
    const int p_add = reverse ? 1 : -2;
    int a1x = static_cast<int>(static_cast<float>(S) * p1.x) + p_add;
    int a1y = static_cast<int>(static_cast<float>(S) * p1.y) + p_add;
    int a2x = static_cast<int>(static_cast<float>(S) * p2.x) - p_add;
    int a2y = static_cast<int>(static_cast<float>(S) * p2.y) - p_add;
    a1x = min(max(a1x, 0), S - 1);
    a1y = min(max(a1y, 0), S - 1);
    a2x = min(max(a2x, 0), S - 1);
    a2y = min(max(a2y, 0), S - 1);
    if (a1y == a2y) return false;
    int ymin = R.vertical ? S - 1 - a1y : S - 1 - a1x;
    int ymax = R.vertical ? S - 1 - a2y : S - 1 - a2x;
    if (reverse) {
        ymin = S - 1 - ymin;
        ymax = S - 1 - ymax;
    }
    if (ymin > ymax) {
        const int t = ymin;
        ymin = ymax;
        ymax = t;
    }
    if (ymin >= ymax) return false;
    R.ymin = ymin;
    R.ymax = ymax;

    const float dir_x = R.ray_x * P.cos_y + R.ray_z * P.sin_y;
    const float dir_y = R.ray_x * P.sin_y - R.ray_z * P.cos_y;
    float sign_x = -1, sign_y = -1;
    R.fix_x = -1;
    R.fix_z = -1;
    float frac_x = P.posx - static_cast<float>(static_cast<int>(P.posx));
    float frac_y = P.posz - static_cast<float>(static_cast<int>(P.posz));
    if (dir_x >= 0) { R.fix_x = 0; sign_x = 1; frac_x = 1 - frac_x; }
    if (dir_y >= 0) { R.fix_z = 0; sign_y = 1; frac_y = 1 - frac_y; }
    D.g0y = dir_y / fabsf(dir_x);
    D.g0x = sign_x;
    D.g1x = dir_x / fabsf(dir_y);
    D.g1y = sign_y;
    D.i0x = D.g0x * frac_x;
    D.i0y = D.g0y * frac_x;
    D.i1x = D.g1x * frac_y;
    D.i1y = D.g1y * frac_y;
    D.gd0 = sqrtf(D.g0x * D.g0x + D.g0y * D.g0y);
    D.gd1 = sqrtf(D.g1x * D.g1x + D.g1y * D.g1y);
    D.dd0 = sqrtf(D.i0x * D.i0x + D.i0y * D.i0y);
    D.dd1 = sqrtf(D.i1x * D.i1x + D.i1y * D.i1y);
    D.dd_now = 0;
    D.pnx = 0;
    D.pny = 0;
    D.index = 0;
    return true;
}

// One DDA cell: the distance along the ray where it begins (it ends where the
// next lane's begins), its level (-1 past the ray's end), its column's index
// there, and the column's table entry.
struct Cell {
    float near;
    int mip;
    uint32_t column;
    uint32_t ex, ey;
};

// Its column's coordinates, x | z << 16, as hit records have them.
__device__ __forceinline__ uint32_t cell_xz(const RayParams& P, const Cell& c) {
    const int shift = P.log2x0 - c.mip;
    return (c.column & ((1u << shift) - 1u)) | ((c.column >> shift) << 16);
}


// A cell's projection: depth and screen numerator of its near edge at column
// index 0, and what its far edge adds.
struct Edge {
    float pz, py, czz, cyy;
};

// Candidate runs a lane records per cell for the merge (shared memory, three
// words per run).  Seven is what three bits count; a cell with more is walked,
// 20 times the cost of a record (six: batches of 64 mixed frames 1.5% slower).
constexpr int kRecs = 7;

// A lane's last coloured sample, stored one pass late: the colour gather
// (a dependent load) then overlaps the following work instead of stalling
// the warp at the store.  Every sample is written once, so the order of
// the stores does not matter.
struct Pending {
    uint32_t* at = nullptr;
    uint32_t colour = 0, z = 0;
    __device__ __forceinline__ void flush() {
        if (at) *at = colour + z;
        at = nullptr;
    }
};

// Per-span constants of the perspective-correct fill (:642-700): screen
// position of the span's far end, texture and 1/z gradients along the span.
struct Span {
    float scr_y1r, u1z, u2dz, onez1, onedz2, umax;
    int texture, sg0;
};

__device__ __forceinline__ Span span_setup(float res_y2, float z_add, float y_add, float pz, float py, float sgs, float sgf,
                                           float tex, int texture) {
    Span sp;
    const float pz1r = pz + z_add * sgs;
    const float py1r = py + y_add * sgs;
    const float pz2r = pz + z_add * sgf;
    const float py2r = py + y_add * sgf;
    const float scr_y2r = res_y2 + py1r / pz1r;
    const float scr_y1r = res_y2 + py2r / pz2r;
    const float u1z = tex / pz2r;
    float u2dz = static_cast<float>(texture) / pz1r - u1z;
    const float onez1 = 1 / pz2r;
    float onedz2 = 1 / pz1r - onez1;
    u2dz /= scr_y2r - scr_y1r;
    onedz2 /= scr_y2r - scr_y1r;
    sp.scr_y1r = scr_y1r;
    sp.u1z = u1z;
    sp.u2dz = u2dz;
    sp.onez1 = onez1;
    sp.onedz2 = onedz2;
    sp.umax = tex - 1.0f;  // a count of colours, below 2^24: exact
    sp.texture = texture;
    sp.sg0 = static_cast<int>(sgs);
    return sp;
}

// Fills samples y .. scr_y2-1 of a span that the occupancy mask leaves open.
template <bool kCount>
__device__ __forceinline__ void draw_span(const Mask& mask, int k, uint32_t* row, float* drow,
                                          rle_hit* hrow, const uint16_t* colours, uint64_t colour_room, int S, int y,
                                          int scr_y2, const Span& sp, int mip, uint32_t vxz, Pending& pend,
                                          Counts& cnt) {
    const float u2dz = sp.u2dz, onedz2 = sp.onedz2;
    if constexpr (kCount) cnt.spans++;
    __syncwarp();  // every lane has read the mask (horizon, y) before any lane claims
    const float mult = static_cast<float>(y + 1) - sp.scr_y1r;
    float uz = sp.u1z + u2dz * mult;
    float onez = sp.onez1 + onedz2 * mult;
    const float umin = static_cast<float>(sp.texture);
    const float umax = sp.umax;
    // 32 pixels per pass: the accumulation runs in lockstep in every lane (it
    // is a chain of IEEE additions, one per sample, masked or not); lane k
    // keeps the values of sample y + k and does its divisions in parallel.
    for (int y0 = y; y0 < scr_y2; y0 += kLanes) {
        const int n = min(kLanes, scr_y2 - y0);
        // lane k needs the accumulators after k more additions
        float my_uz = uz, my_onez = onez;
        for (int j = 0; j < k && j < n; j++) {
            my_uz += u2dz;
            my_onez += onedz2;
        }
        if (n == kLanes) {  // start of the next pass: 32 additions from this one
            uz = __shfl_sync(kWarp, my_uz, kLanes - 1) + u2dz;
            onez = __shfl_sync(kWarp, my_onez, kLanes - 1) + onedz2;
        }
        const int yy = y0 + k;
        bool wrote = false;
        if (yy < scr_y2 && !mask.get(yy) && in_bounds(yy < S, kBoundsRay, static_cast<unsigned long long>(yy))) {
            const uint32_t u = static_cast<uint32_t>(fminf(fmaxf(my_uz / my_onez, umin), umax));
            const float depth = 1 / my_onez;
            const uint32_t real_z = static_cast<uint32_t>(static_cast<int>(depth) & 0xfffe);
            pend.flush();
            pend.at = &row[yy];
            pend.colour = in_bounds(u < colour_room, kBoundsColour, u) ? __ldg(&colours[u]) : 0u;
            pend.z = real_z << 16;
            drow[yy] = depth;
            if (hrow) {
                rle_hit h;
                h.x = static_cast<uint16_t>(vxz & 0xffffu);
                h.z = static_cast<uint16_t>(vxz >> 16);
                h.y = static_cast<uint16_t>((sp.sg0 >> mip) + static_cast<int>(u - static_cast<uint32_t>(sp.texture)));
                h.mip = static_cast<uint8_t>(mip);
                h.flags = 1;
                hrow[yy] = h;
            }
            atomicOr(&mask.w[yy >> 5], 1u << (yy & 31));
            wrote = true;
        }
        if constexpr (kCount) cnt.pixels += __popc(__ballot_sync(kWarp, wrote));
        __syncwarp();
    }
}

// Exact sequential processing of one cell (the body of the reference's main
// loop after the DDA step).  Uniform across the warp.
template <bool kCount>
__device__ __forceinline__ void merge_cell(const RayParams& P, const Ray& R, const Mask& mask, int k,
                                           uint32_t* row, float* drow, rle_hit* hrow, const Cell& c, const Edge& e, int& ymin,
                                           int& ymax, Counts& cnt) {
    const float res_y2 = static_cast<float>(P.S / 2);
    Pending pend;
    // clip top (:467)
    if (e.pz * res_y2 + e.py <= e.pz * static_cast<float>(ymin)) return;
    if constexpr (kCount) cnt.fetched++;
    const uint16_t* hdr = P.slabs[c.mip] + 2 + c.ex;
    const int nruns = c.ey & 0xffffu;
    const uint16_t* colours = hdr + nruns;
    const float mountain = P.posy;
    uint32_t sti = c.ey >> 16;
    int sg = 0;
    float tex = 0;
    for (int r = 0; r < nruns; r++) {
        if (r > 0) {
            const uint64_t hi = static_cast<uint64_t>(c.ex) + 2u + static_cast<uint64_t>(r);
            sti = in_bounds(hi < P.slab_words[c.mip], kBoundsHeader, hi) ? __ldg(&hdr[r]) : 0u;
            if constexpr (kCount) cnt.headers++;
        }
        int solid = static_cast<int>(sti >> 10);
        sg += static_cast<int>(sti & 1023u) << c.mip;
        if (solid == 0) continue;
        const int texture = static_cast<int>(tex);
        tex += static_cast<float>(solid);
        solid <<= c.mip;
        const float sgs = static_cast<float>(sg);
        sg += solid;
        const float sgf = static_cast<float>(sg);
        if constexpr (kCount) cnt.runs++;
        float czz1 = e.pz, cyy1 = e.py;
        if (mountain + sgs >= 0) { czz1 += e.czz; cyy1 += e.cyy; }
        const float pz1 = czz1 + R.pos3d_z_add * sgs;
        if (pz1 <= 0) continue;
        const float py1 = cyy1 + R.pos3d_y_add * sgs;
        int scr_y2 = static_cast<int>(res_y2 + py1 / pz1);
        if (scr_y2 <= ymin) break;
        float czz2 = e.pz, cyy2 = e.py;
        if (mountain + sgf < 0) { czz2 += e.czz; cyy2 += e.cyy; }
        const float pz2 = czz2 + R.pos3d_z_add * sgf;
        if (pz2 <= 0) continue;
        const float py2 = cyy2 + R.pos3d_y_add * sgf;
        int scr_y1 = static_cast<int>(res_y2 + py2 / pz2 - 1);
        if (scr_y1 >= ymax) continue;
        // floating horizon (:563-580)
        if (scr_y2 >= ymax) {
            scr_y2 = ymax;
            ymax = scr_y1;
        }
        if (scr_y1 <= ymin) {
            scr_y1 = ymin;
            ymin = scr_y2;
            ymin = mask.first_clear(ymin, ymax > ymin ? ymax : ymin);
        }
        const int y = mask.first_clear(scr_y1, scr_y2);
        if (y >= scr_y2) continue;
        const Span sp = span_setup(res_y2, R.pos3d_z_add, R.pos3d_y_add, e.pz, e.py, sgs, sgf, tex, texture);
        const uint64_t cofs = static_cast<uint64_t>(c.ex) + 2u + static_cast<uint64_t>(nruns);
        const uint64_t room = cofs <= P.slab_words[c.mip] ? P.slab_words[c.mip] - cofs : 0u;
        draw_span<kCount>(mask, k, row, drow, hrow, colours, room, P.S, y, scr_y2, sp, c.mip, cell_xz(P, c),
                             pend, cnt);
    }
    pend.flush();
}


// Where the DDA of one ray stands between chunks (uniform in its warp).
struct Walk {
    Dda d;        // (dd_now, pnx, pny, index: the last event, right in the last lane at least)
    DdaCache c;   // steps of d's chains, while `cached`
    bool cached;
    int room;     // steps that need no check for a LOD switch or the ray's end
    float z, dz, zswitch;
    int mapswitch, mip;
};

// Level-of-detail switch at the top of a step (:343-365): past the switch
// distance the ray moves to the next mip level and doubles its step.
__device__ __forceinline__ void lod_switch(Walk& w, int nummaps) {
    while (w.z > w.zswitch) {
        if (w.mip < nummaps - 1) w.mip++;
        w.d.g0x *= 2; w.d.g0y *= 2; w.d.g1x *= 2; w.d.g1y *= 2;
        w.d.gd0 *= 2; w.d.gd1 *= 2;
        w.mapswitch *= 2;
        w.zswitch = static_cast<float>(w.mapswitch);
        w.dz *= 2;
    }
}

// What a DDA step gives for its cell.
struct ChunkStep {
    float near, pbx, pby;
    int ib, mip;
};

// The cell of one DDA step.  Its table entry is loaded at the top of its own
// turn of the chunk loop, under the next chunk's DDA: loaded a turn earlier, its
// registers are waited for where the loop hands them on, which was a sixth of
// a slow ray's time (1920x1080 frames 313 -> 279 us; staged in L1 or L2 a turn
// earlier as well: no gain, nor through asynchronous copies to shared memory).
__device__ __forceinline__ Cell cell_of_step(const RayParams& P, const Ray& R, bool valid, const ChunkStep& st) {
    const int voxel_x = static_cast<int>(P.posx + st.pbx) + (st.ib ? 0 : R.fix_x);
    const int voxel_z = static_cast<int>(P.posz + st.pby) + (st.ib ? R.fix_z : 0);
    const uint32_t vx = static_cast<uint32_t>(voxel_x & (P.gridx0 - 1)) >> st.mip;
    const uint32_t vz = static_cast<uint32_t>(voxel_z & (P.gridz0 - 1)) >> st.mip;
    Cell c;
    c.near = st.near;
    c.mip = valid ? st.mip : -1;
    c.column = vx + (vz << (P.log2x0 - st.mip));
    return c;
}

__device__ __forceinline__ uint2 cell_entry(const RayParams& P, const Cell& c) {
    return c.mip >= 0 && in_bounds(c.column < P.table_cols[c.mip], kBoundsTable, c.column)
               ? __ldg(&P.table[c.mip][c.column])
               : make_uint2(0u, 0u);
}

__device__ __forceinline__ Edge cell_edge(const RayParams& P, const Ray& R, float near, float far) {
    const float sin_x = P.sin_x, cos_x = P.cos_x;
    const float mountain = P.posy;
    const float delta = far - near;
    const float vs_x = R.ray_x * near;
    const float vs_z = R.ray_z * near;
    const float corr_x = R.ray_x * delta;
    const float corr_z = R.ray_z * delta;
    Edge e;
    e.pz = cos_x * vs_z + sin_x * mountain;
    const float py = R.vertical ? cos_x * mountain - sin_x * vs_z : vs_x;
    e.py = py * R.rmul;
    e.czz = cos_x * corr_z;
    const float cyy = R.vertical ? -sin_x * corr_z : corr_x;
    e.cyy = cyy * R.rmul;
    return e;
}

// Pre-culls a cell against the horizon at the start of its chunk and scans
// its runs.  Returns the number of runs recorded in `rec` (one slot every
// `stride` entries) that the exact walk could still draw, or -1 if the cell
// has to be walked run by run at its turn.  Run headers are loaded two runs
// ahead (the first travels in the table entry).
//
// A run is recorded unless, at the chunk's horizon, the walk would skip it for
// good (`pz1 <= 0`, `pz2 <= 0`, `scr_y1 >= ymax`) or none of its samples in the
// open range [ymin, ymax) is still free in the occupancy mask: the mask only
// gains bits and the range only closes.  The scan ends where the walk would
// already break at the chunk's horizon (`scr_y2 <= ymin`).
//
// What a recorded cell draws depends only on which of its samples are free at
// its turn, not on the horizon then: ymin always names the first free sample
// (or the range is closed), so a span that reaches it starts with a free
// sample, and the ymax a span sets cuts off samples that are all taken.  The
// walk's two tests that stop a cell by the horizon alone agree with that
// under two conditions, checked here; a cell that fails one is walked:
//  * the break test at a run drops that run and all later ones.  If no later
//    recorded run reaches higher than any run before it, a break means that
//    none of them has a free sample left;
//  * the clip-top test at the cell drops all of it.  It must stay false up to
//    the last horizon at which a recorded run still has a sample above it
//    (for pz >= 0 it gets truer as ymin grows, for pz < 0 less true).
__device__ __forceinline__ int scan_runs(const RayParams& P, const Ray& R, const Mask& mask, int ymin, int ymax,
                                         const Cell& c, const Edge& e, uint32_t* rec, int stride) {
    const float res_y2 = static_cast<float>(P.S / 2);
    const float mountain = P.posy;
    const int mip = c.mip;
    // clip top at the current horizon
    if (e.pz >= 0.0f && e.pz * res_y2 + e.py <= e.pz * static_cast<float>(ymin)) return 0;
    const int nruns = c.ey & 0xffffu;
    const uint16_t* hdr = P.slabs[mip] + 2 + c.ex;
    auto header = [&](int r) -> uint32_t {
        const uint64_t hi = static_cast<uint64_t>(c.ex) + 2u + static_cast<uint64_t>(r);
        return r < nruns && in_bounds(hi < P.slab_words[mip], kBoundsHeader, hi) ? __ldg(&hdr[r]) : 0u;
    };
    uint32_t sti = c.ey >> 16, next = header(1), after = header(2);
    int sg = 0, texi = 0, n = 0;
    int low = 0x7fffffff;  // lowest reach (scr_y2) of the runs so far
    int top = 0;           // end of the highest recorded span
    for (int r = 0; r < nruns; r++) {
        const int solid = static_cast<int>(sti >> 10);
        sg += static_cast<int>(sti & 1023u) << mip;
        sti = next;
        next = after;
        after = header(r + 3);
        if (solid == 0) continue;
        const int texture = texi, start = sg;
        texi += solid;
        const float sgs = static_cast<float>(sg);
        sg += solid << mip;
        const float sgf = static_cast<float>(sg);
        float czz1 = e.pz, cyy1 = e.py;
        if (mountain + sgs >= 0) { czz1 += e.czz; cyy1 += e.cyy; }
        const float pz1 = czz1 + R.pos3d_z_add * sgs;
        if (pz1 <= 0) continue;
        const float py1 = cyy1 + R.pos3d_y_add * sgs;
        const int scr_y2 = static_cast<int>(res_y2 + py1 / pz1);
        if (scr_y2 <= ymin) break;  // the walk breaks here or earlier
        low = min(low, scr_y2);
        float czz2 = e.pz, cyy2 = e.py;
        if (mountain + sgf < 0) { czz2 += e.czz; cyy2 += e.cyy; }
        const float pz2 = czz2 + R.pos3d_z_add * sgf;
        if (pz2 <= 0) continue;
        const float py2 = cyy2 + R.pos3d_y_add * sgf;
        const int scr_y1 = static_cast<int>(res_y2 + py2 / pz2 - 1);
        if (scr_y1 >= ymax) continue;
        const int hi = min(scr_y2, ymax);
        const int lo = mask.first_clear(max(scr_y1, ymin), hi);
        if (lo >= hi) continue;  // every sample it could colour is taken already
        if (n == kRecs || scr_y2 != low) return -1;
        rec[(3 * n) * stride] = static_cast<uint32_t>(lo) | (static_cast<uint32_t>(hi) << 16);
        rec[(3 * n + 1) * stride] = static_cast<uint32_t>(start);
        rec[(3 * n + 2) * stride] = static_cast<uint32_t>(texture) | (static_cast<uint32_t>(solid) << 16);
        top = max(top, hi);
        n++;
    }
    if (n > 0) {
        const int t = e.pz >= 0.0f ? top - 1 : ymin;
        if (e.pz * res_y2 + e.py <= e.pz * static_cast<float>(t)) return -1;
    }
    return n;
}

// Spans are not filled when their turn comes: their free samples are claimed
// in the occupancy mask and queued in pieces, one per mask word; a flush then
// colours the samples of up to 32 pieces 32 at a time, one sample per lane.
// Queue entry: 2 x uint4 in shared memory, vector v of entry e at [32 * v + e],
//   {y0 | p0 << 14 | level << 28, claimed samples as bits from p0,
//    colour offset of the column, texture | colours << 16},
//   {pz, py, start of the run on the column axis, vx | vz << 16}
// with y0 the span's first claimed sample, where its accumulation starts, and
// p0 the piece's (sample indexes are below 2^14, a column holds fewer than
// 2^16 colours and a run at most 63, so the fields fit).  The constants of
// the fill (8 divisions) are formed by the lane that holds an entry in the
// flush, for up to 32 pieces at once, and replace the second vector.
constexpr int kQueueVecs = 2;

struct SpanQueue {
    uint4* e;  // 32 entries of this ray
    int n;
};

// Position of the set bit number r (from 0) of m, which has more than r bits.
__device__ __forceinline__ int nth_bit(uint32_t m, int r) {
    if ((m & (m + 1u)) == 0u) return r;  // 0..01..1: most spans are claimed whole
    int at = 0;
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) {
        const int low = __popc(m & ((1u << w) - 1u));
        if (r >= low) {
            r -= low;
            at += w;
            m >>= w;
        }
    }
    return at;
}

__device__ __forceinline__ void flush_spans(const RayParams& P, float z_add, float y_add, uint4* queue, int n, int k,
                                            uint32_t* row, float* drow, rle_hit* hrow) {
    Pending pend;
    uint4 e0 = make_uint4(0u, 0u, 0u, 0u), e1 = e0;
    if (k < n) {
        e0 = queue[k];
        e1 = queue[kLanes + k];
    }
    // samples per queued piece, inclusive prefix over the lanes
    const int cnt = __popc(e0.y);
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < kLanes; o <<= 1) {
        const int v = __shfl_up_sync(kWarp, incl, o);
        if (k >= o) incl += v;
    }
    const int total = __shfl_sync(kWarp, incl, n - 1);
    const int start = incl - cnt;
    // this lane's piece: the accumulators at its first sample and their step,
    // rounded (the sums are then one multiply-add away) or, where they leave
    // their binade within the piece, as it is
    if (k < n) {
        const int sg = static_cast<int>(e1.z), texture = static_cast<int>(e0.w & 0xffffu);
        const int solid = static_cast<int>(e0.w >> 16), mip = static_cast<int>(e0.x >> 28);
        const Span sp = span_setup(static_cast<float>(P.S / 2), z_add, y_add, __uint_as_float(e1.x), __uint_as_float(e1.y),
                                   static_cast<float>(sg), static_cast<float>(sg + (solid << mip)),
                                   static_cast<float>(texture + solid), texture);
        const int y0 = static_cast<int>(e0.x & 0x3fffu), skip = static_cast<int>((e0.x >> 14) & 0x3fffu) - y0;
        const float mult = static_cast<float>(y0 + 1) - sp.scr_y1r;
        const float uz = accumulate(sp.u1z + sp.u2dz * mult, sp.u2dz, skip);
        const float onez = accumulate(sp.onez1 + sp.onedz2 * mult, sp.onedz2, skip);
        const int steps = 31 - __clz(static_cast<int>(e0.y));  // to the piece's last claimed sample
        float du, dz;
        const bool jump = steady_step(uz, sp.u2dz, steps, &du) & steady_step(onez, sp.onedz2, steps, &dz);
        queue[k].x = e0.x | (jump ? 0x80000000u : 0u);
        queue[kLanes + k] = make_uint4(bits_of(uz), bits_of(jump ? du : sp.u2dz), bits_of(onez),
                                bits_of(jump ? dz : sp.onedz2));
    }
    __syncwarp();
    for (int b = 0; b < total; b += kLanes) {
        const int t = b + k;
        // piece of sample t: entries start at strictly increasing sample
        // numbers (every queued piece owns at least one sample); those that
        // start at or before b, plus those starting in (b, b + k], count
        // the pieces at or before t
        const bool entry = k < n;
        unsigned le = __ballot_sync(kWarp, entry && start <= b);
        const unsigned marks =
            __reduce_or_sync(kWarp, (entry && start > b && start < b + kLanes) ? (1u << (start - b)) : 0u);
        const unsigned upto = k >= 31 ? 0xffffffffu : ((2u << k) - 1u);
        const int from = __popc(le) - 1 + __popc(marks & upto);
        const int before = __shfl_sync(kWarp, start, from);
        uint32_t vxz = 0, sg = 0;
        if (hrow) {
            vxz = __shfl_sync(kWarp, e1.w, from);
            sg = __shfl_sync(kWarp, e1.z, from);
        }
        if (t < total) {
            const uint4 v0 = queue[from], v1 = queue[kLanes + from];
            const uint32_t at = v0.x, cofs = v0.z, tc = v0.w;
            const int mip = static_cast<int>((at >> 28) & 7u);
            const int steps = nth_bit(v0.y, t - before);
            const int p = static_cast<int>((at >> 14) & 0x3fffu) + steps;
            float uz = __uint_as_float(v1.x), onez = __uint_as_float(v1.z);
            if (at & 0x80000000u) {
                uz = __fmaf_rn(static_cast<float>(steps), __uint_as_float(v1.y), uz);
                onez = __fmaf_rn(static_cast<float>(steps), __uint_as_float(v1.w), onez);
            } else {
                for (int j = 0; j < steps; j++) {
                    uz += __uint_as_float(v1.y);
                    onez += __uint_as_float(v1.w);
                }
            }
            const int texture = static_cast<int>(tc & 0xffffu);
            const float umax = static_cast<float>(texture + static_cast<int>(tc >> 16) - 1);
            const uint32_t u = static_cast<uint32_t>(fminf(fmaxf(uz / onez, static_cast<float>(texture)), umax));
            const float depth = 1 / onez;
            const uint32_t real_z = static_cast<uint32_t>(static_cast<int>(depth) & 0xfffe);
            const uint64_t ci = static_cast<uint64_t>(cofs) + u;
            if (in_bounds(p < P.S, kBoundsRay, static_cast<unsigned long long>(p))) {
                pend.flush();
                pend.at = &row[p];
                pend.colour = in_bounds(ci < P.slab_words[mip], kBoundsColour, ci) ? __ldg(&P.slabs[mip][ci]) : 0u;
                pend.z = real_z << 16;
                drow[p] = depth;
            }
            if (hrow && p < P.S) {
                rle_hit h;
                h.x = static_cast<uint16_t>(vxz & 0xffffu);
                h.z = static_cast<uint16_t>(vxz >> 16);
                const int sg0 = static_cast<int>(static_cast<float>(static_cast<int>(sg)));
                h.y = static_cast<uint16_t>((sg0 >> mip) + static_cast<int>(u - static_cast<uint32_t>(texture)));
                h.mip = static_cast<uint8_t>(mip);
                h.flags = 1;
                hrow[p] = h;
            }
        }
    }
    pend.flush();
    __syncwarp();  // the entries are rewritten by the next spans
}

// ~0 << max(n, 0), 0 from n = 32 on: the samples at or past place n of a
// 32-sample window.
__device__ __forceinline__ uint32_t from_place(int n) {
    uint32_t r;
    asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(0xffffffffu), "r"(max(n, 0)));
    return r;
}

// The cell of lane `from`, and its projection, in every lane.
__device__ __forceinline__ Cell cell_of(const Cell& c, int from) {
    Cell r;
    r.near = 0.0f;  // in the projection
    r.ex = __shfl_sync(kWarp, c.ex, from);
    r.ey = __shfl_sync(kWarp, c.ey, from);
    r.mip = __shfl_sync(kWarp, c.mip, from);
    r.column = __shfl_sync(kWarp, c.column, from);
    return r;
}
__device__ __forceinline__ Edge edge_of(const Edge& e, int from) {
    Edge r;
    r.pz = __shfl_sync(kWarp, e.pz, from);
    r.py = __shfl_sync(kWarp, e.py, from);
    r.czz = __shfl_sync(kWarp, e.czz, from);
    r.cyy = __shfl_sync(kWarp, e.cyy, from);
    return r;
}

// Draws what the lanes' scans recorded, in the order of the sequential walk
// (cell by cell, run by run): every sample goes to the first span that covers
// it and finds it free.  The chunk's records, numbered in that order, go one
// to a lane; then, for each word of the occupancy mask that they reach, an OR
// over the lanes before its own tells a lane which of its samples earlier
// spans cover.  What is left of its span in the word, and free, it queues.  A
// cell that has to be walked is a barrier: the records before it are claimed
// first, then the warp walks it.
//
// Bound by latency and issue: a frame ends with its slowest ray, and the
// sequential form of this step (one record after another, two or three
// dependent shared-memory loads and a queue insert each; spans of more than
// 32 samples filled one at a time) took half of that ray: 1920x1080 frames 466
// -> 438 us and 3840x2160 frames 424 -> 336 us without it.  A prefix OR takes
// five shuffles per word where one lane after another took 80 cycles per span
// (4700 -> 3000 cycles per chunk that draws; 1920x1080 frames 350 -> 310 us).
__device__ __forceinline__ void merge_chunk(const RayParams& P, const Ray& R, const Mask& mask, int k,
                                            uint32_t* row, float* drow, rle_hit* hrow, const Cell& c, const Edge& edge,
                                            int nrec, const uint32_t* warp_recs, int stride, uint32_t* list, int& ymin,
                                            int& ymax, SpanQueue& q, Counts& cnt) {
    // entries before this lane's cell, and in all: its records (at most kRecs,
    // three bits), or one for a cell to walk
    const int mine = nrec < 0 ? 1 : nrec;
    const unsigned n0 = __ballot_sync(kWarp, mine & 1), n1 = __ballot_sync(kWarp, mine & 2),
                   n2 = __ballot_sync(kWarp, mine & 4);
    const unsigned lt = (1u << k) - 1u;
    const int base = __popc(n0 & lt) + 2 * __popc(n1 & lt) + 4 * __popc(n2 & lt);
    const int total = __popc(n0) + 2 * __popc(n1) + 4 * __popc(n2);
    for (int first = 0; first < total; first += kLanes) {
        const int n = min(kLanes, total - first);
        // list[i] = lane | record << 5 of entry i, or a cell to walk
        for (int r = 0; r < mine; r++) {
            const int at = base + r - first;
            if (at >= 0 && at < kLanes) list[at] = static_cast<uint32_t>(k) | (r << 5) | (nrec < 0 ? 0x100u : 0u);
        }
        __syncwarp();  // the list and the records are read by the whole warp
        const uint32_t entry = k < n ? list[k] : 0u;
        const int src = k < n ? static_cast<int>(entry & 31u) : 0;
        const bool walk = (entry & 0x100u) != 0u;
        uint32_t range = 0u, begin = 0u, colours = 0u;
        if (k < n && !walk) {
            const uint32_t* rec = warp_recs + 3 * static_cast<int>((entry >> 5) & 7u) * stride + src;
            range = rec[0];
            begin = rec[stride];
            colours = rec[2 * stride];
        }
        const int lo = static_cast<int>(range & 0xffffu), hi = static_cast<int>(range >> 16);
        const float pz = __shfl_sync(kWarp, edge.pz, src), py = __shfl_sync(kWarp, edge.py, src);
        const int mip = __shfl_sync(kWarp, c.mip, src);
        const uint32_t cofs = __shfl_sync(kWarp, c.ex + 2u + (c.ey & 0xffffu), src);
        uint32_t vxz = 0;
        if (hrow) vxz = __shfl_sync(kWarp, cell_xz(P, c), src);
        unsigned walks = __ballot_sync(kWarp, walk);
        int start = 0;
        for (;;) {
            const int stop = walks ? __ffs(walks) - 1 : n;
            if (stop > start) {
                // ---- spans [start, stop): claim the free samples ----
                const bool in = k >= start && k < stop;
                const int from = static_cast<int>(__reduce_min_sync(kWarp, in ? static_cast<unsigned>(lo) : ~0u)) & ~31;
                const int to = static_cast<int>(__reduce_max_sync(kWarp, in ? static_cast<unsigned>(hi) : 0u));
                int y0 = -1;  // the span's first claimed sample
                for (int w = from; w < to; w += 32) {
                    const uint32_t taken = mask.w[w >> 5];
                    if (taken == 0xffffffffu) continue;
                    const uint32_t bits = in ? from_place(lo - w) & ~from_place(hi - w) : 0u;
                    // the first span here, and whether it alone counts: it covers the
                    // word, or no other span reaches it (the inside of long spans)
                    const unsigned reach = __ballot_sync(kWarp, bits != 0u);
                    const unsigned whole = __ballot_sync(kWarp, bits == 0xffffffffu);
                    uint32_t own = bits & ~taken, all;
                    if ((reach & (reach - 1u)) == 0u || (whole & reach & (0u - reach)) != 0u) {
                        const int f = __ffs(reach) - 1;
                        all = __shfl_sync(kWarp, bits, max(f, 0));
                        if (k != f) own = 0u;
                    } else {
                        uint32_t before = __shfl_up_sync(kWarp, bits, 1);
                        if (k == 0) before = 0u;
#pragma unroll
                        for (int o = 1; o < kLanes; o <<= 1) {
                            const uint32_t v = __shfl_up_sync(kWarp, before, o);
                            if (k >= o) before |= v;
                        }
                        own &= ~before;
                        all = __reduce_or_sync(kWarp, bits);
                    }
                    const unsigned claims = __ballot_sync(kWarp, own != 0u);
                    if (!claims) continue;
                    mask.w[w >> 5] = taken | all;  // by every lane, the same word
                    const int m = __popc(claims);
                    if (q.n + m > kLanes) {
                        flush_spans(P, R.pos3d_z_add, R.pos3d_y_add, q.e, q.n, k, row, drow, hrow);
                        q.n = 0;
                    }
                    if (own) {
                        const int skip = __ffs(own) - 1, p0 = w + skip;
                        if (y0 < 0) y0 = p0;
                        uint4* e = q.e + q.n + __popc(claims & ((1u << k) - 1u));
                        e[0] = make_uint4(static_cast<uint32_t>(y0) | (static_cast<uint32_t>(p0) << 14) |
                                              (static_cast<uint32_t>(mip) << 28),
                                          own >> skip, cofs, colours);
                        e[kLanes] = make_uint4(__float_as_uint(pz), __float_as_uint(py), begin, vxz);
                    }
                    q.n += m;
                    __syncwarp();
                }
                __syncwarp();  // the mask's words
                ymin = mask.first_clear(ymin, max(ymin, ymax));
                if (to >= ymax) ymax = mask.last_clear(ymin, ymax);
            }
            if (stop >= n || ymin >= ymax) break;
            // ---- a cell to walk ----
            walks &= walks - 1;
            start = stop + 1;
            const int from = __shfl_sync(kWarp, src, stop);
            merge_cell<false>(P, R, mask, k, row, drow, hrow, cell_of(c, from),
                                 edge_of(edge, from), ymin, ymax, cnt);
            if (start >= n || ymin >= ymax) break;
        }
        __syncwarp();  // the list and the records are rewritten
        if (ymin >= ymax) return;
    }
}

// Steps from here that can meet neither a LOD switch nor the end of the ray.
// z, dz (a power of two) and the switch distances are whole numbers held in
// floats, exactly below 2^24.
__device__ __forceinline__ int steps_unchecked(const RayParams& P, const Walk& W) {
    if (!dda_can_jump(W.d) || !(W.z + W.dz < 16777216.0f)) return 0;
    const int zi = static_cast<int>(W.z), shift = 31 - __clz(static_cast<int>(W.dz));
    const int to_switch = W.mapswitch - zi, to_end = min(P.z_far, 16777216) - zi;
    return to_switch < 0 || to_end < 0 ? 0 : min((to_switch >> shift) + 1, to_end >> shift);
}

// One chunk of the DDA: lane k's cell is that of step k, from the event of
// step k and that of the step before (a shuffle from lane k-1; lane 0 takes
// the last event of the chunk before).  Advances W past the chunk and returns
// how many of its steps are valid (fewer than 32: the ray ends).
//
// Lane k finds the event of step k without the k steps before it (dda_jump).
// Usually all lanes do, and the chunk is one straight line with the chains'
// steps kept from the chunk before.  Where a chain leaves its binade, the
// lanes up to there are done, the state goes one plain step on and the rest
// jump again; a chain leaves its binade when the distance doubles, which is
// one chunk in three (of 30) to one in seven (of 200).  LOD switches and the
// ray's end cut a chunk the same way.  The ray's first chunk, where distances
// double most, takes plain steps.
//
// Bound by latency and issue: in lockstep, 32 steps of 22 instructions each,
// repeated by every lane, were 700 of a chunk's 860 instructions.  Together
// with the horizon test that drops whole chunks before they are projected
// (cell_alive) and the word-wise merge, per frame: 1920x1080 438 -> 310 us,
// 1366x768 with hits 278 -> 225 us, 640x480 152 -> 130 us, 320x240 87 -> 82 us.
__device__ __forceinline__ int dda_chunk(const RayParams& P, Walk& W, int k, ChunkStep& st) {
    const float start_dd = W.d.dd_now, start_px = W.d.pnx, start_py = W.d.pny;
    const int start_ix = W.d.index;
    float c_dd = 0, c_px = 0, c_py = 0;
    int c_ix = 0, smip = W.mip;
    int nvalid = kLanes;
    int pos = 0;  // steps taken
    int jumps = W.z == 0.0f ? 0 : 3;
    if (W.cached && W.room >= kLanes) {
        const DdaJump j = dda_jump(W.d, W.c, static_cast<float>(k));
        const unsigned bad = __ballot_sync(kWarp, !j.ok);
        const unsigned kept = __ballot_sync(kWarp, j.kept);
        float dd0 = __shfl_sync(kWarp, j.dd0, kLanes - 1), dd1 = __shfl_sync(kWarp, j.dd1, kLanes - 1);
        float i0x = __shfl_sync(kWarp, j.i0x, kLanes - 1), i0y = __shfl_sync(kWarp, j.i0y, kLanes - 1);
        float i1x = __shfl_sync(kWarp, j.i1x, kLanes - 1), i1y = __shfl_sync(kWarp, j.i1y, kLanes - 1);
        c_dd = j.dd;
        c_px = j.px;
        c_py = j.py;
        c_ix = j.axis1 ? 1 : 0;
        pos = kLanes;
        W.cached = kept >> 31;
        if (bad) {  // up to the lane that is the first out of place; its event is right
            pos = __ffs(bad);
            const int src = max(pos - 2, 0);
            dd0 = __shfl_sync(kWarp, j.dd0, src);
            dd1 = __shfl_sync(kWarp, j.dd1, src);
            i0x = __shfl_sync(kWarp, j.i0x, src);
            i0y = __shfl_sync(kWarp, j.i0y, src);
            i1x = __shfl_sync(kWarp, j.i1x, src);
            i1y = __shfl_sync(kWarp, j.i1y, src);
            W.cached = false;
        }
        if (pos > 1) {
            W.d.dd0 = dd0;
            W.d.dd1 = dd1;
            W.d.i0x = i0x;
            W.d.i0y = i0y;
            W.d.i1x = i1x;
            W.d.i1y = i1y;
        }
        if (bad) dda_step(W.d);
        W.z += W.dz * static_cast<float>(pos);
        W.room -= pos;
        jumps = 2;
    }
    if (pos < kLanes) {
        const float zfar = static_cast<float>(P.z_far);
#pragma unroll 1
        while (pos < kLanes) {
            const int lim = min(kLanes, pos + W.room);
            if (W.room > 0 && jumps > 0) {
                jumps--;
                if (!W.cached) W.c = dda_cache(W.d);
                const DdaJump j = dda_jump(W.d, W.c, static_cast<float>(max(k - pos, 0)));
                const unsigned bad = __ballot_sync(kWarp, k >= pos && !j.ok);
                const unsigned kept = __ballot_sync(kWarp, j.kept);
                const int stop = min(bad ? __ffs(bad) - 1 : kLanes, lim);
                if (k >= pos && k <= stop && k < lim) {
                    c_dd = j.dd;
                    c_px = j.px;
                    c_py = j.py;
                    c_ix = j.axis1 ? 1 : 0;
                }
                W.cached = true;
                if (stop > pos) {
                    const int src = stop - 1;
                    W.d.dd0 = __shfl_sync(kWarp, j.dd0, src);
                    W.d.i0x = __shfl_sync(kWarp, j.i0x, src);
                    W.d.i0y = __shfl_sync(kWarp, j.i0y, src);
                    W.d.dd1 = __shfl_sync(kWarp, j.dd1, src);
                    W.d.i1x = __shfl_sync(kWarp, j.i1x, src);
                    W.d.i1y = __shfl_sync(kWarp, j.i1y, src);
                    W.cached = (kept >> (stop - 1)) & 1u;
                }
                int taken = stop - pos;
                if (stop < lim) {
                    dda_step(W.d);
                    W.cached = false;
                    taken++;
                }
                W.z += W.dz * static_cast<float>(taken);
                W.room -= taken;
                pos += taken;
            } else if (W.room > 0) {
                W.z += W.dz * static_cast<float>(lim - pos);
                W.room -= lim - pos;
                W.cached = false;
#pragma unroll 1
                for (; pos < lim; pos++) {
                    dda_step(W.d);
                    if (pos == k) {
                        c_dd = W.d.dd_now;
                        c_px = W.d.pnx;
                        c_py = W.d.pny;
                        c_ix = W.d.index;
                    }
                }
            } else {
                if (W.z > W.zswitch) {
                    lod_switch(W, P.nummaps);
                    if (k >= pos) smip = W.mip;  // cells from this step on use the new level
                }
                W.z += W.dz;
                if (W.z > zfar) {
                    nvalid = pos;
                    break;
                }
                dda_step(W.d);
                if (pos == k) {
                    c_dd = W.d.dd_now;
                    c_px = W.d.pnx;
                    c_py = W.d.pny;
                    c_ix = W.d.index;
                }
                pos++;
                W.cached = false;
                W.room = steps_unchecked(P, W);
            }
        }
    }
    // the last event, for the next chunk's first cell
    if (k == kLanes - 1) {
        W.d.dd_now = c_dd;
        W.d.pnx = c_px;
        W.d.pny = c_py;
        W.d.index = c_ix;
    }
    // lane k takes lane k-1's values and lane 0 those that the last lane had
    // at the start of the chunk
    const int prev = (k + kLanes - 1) % kLanes;
    const bool last = k == kLanes - 1;
    st.near = __shfl_sync(kWarp, last ? start_dd : c_dd, prev);
    st.pbx = __shfl_sync(kWarp, last ? start_px : c_px, prev);
    st.pby = __shfl_sync(kWarp, last ? start_py : c_py, prev);
    st.ib = __shfl_sync(kWarp, last ? start_ix : c_ix, prev);
    st.mip = smip;
    return nvalid;
}

// What can still be drawn above the horizon ymin, as a bound that a cell is
// tested against before anything of it is projected.
//
// A run whose top lies h below the eye (h = position.y + its column index,
// level-0 units, h grows downwards) seen at distance t projects with
// pz1 = c*t + d*h and py1 = py_t*t + py_h*h (c = cos_x*ray_z, d = sin_x;
// py_t = -rmul*sin_x*ray_z, py_h = rmul*cos_x for rays of the up/down fans,
// py_t = rmul*ray_x, py_h = 0 for the left/right fans; :483-559).  The run is
// dropped at its turn (`scr_y2 <= ymin`, or `pz1 <= 0`) whenever
// f = K*pz1 + py1 < 0 with K = res_y2 - ymin - 1.  f = a*t + b*h is linear, so
// where its slope in h is not positive, f < 0 at a column's topmost run and at
// the end of the cell where f is larger drops all of the column; and where
// its slope in t is not positive either, f < 0 at the scene's topmost voxel
// drops all cells from t on.  A margin of 1e-4 of the magnitudes of the terms
// covers the float rounding of the kernel's evaluation (about 1e-6 relative);
// ymin only grows later, which only lowers f where pz1 > 0.
struct Horizon {
    float a, b, eb;  // bound of f: a*t + b*h + eb*|h|
    float scene;     // b*h + eb*|h| of the scene's topmost voxel, or +inf
};

__device__ __forceinline__ Horizon horizon_bound(const RayParams& P, const Ray& R, int ymin) {
    const float eps = 1e-4f;
    const float res_y2 = static_cast<float>(P.S / 2);
    const float K = res_y2 - static_cast<float>(ymin) - 1.0f;
    const float c = P.cos_x * R.ray_z, d = P.sin_x;
    const float py_t = R.vertical ? -R.rmul * P.sin_x * R.ray_z : R.rmul * R.ray_x;
    const float py_h = R.vertical ? R.rmul * P.cos_x : 0.0f;
    const float scale = res_y2 + fabsf(K) + 1.0f;
    const float ma = fabsf(c) * scale + fabsf(py_t), mb = fabsf(d) * scale + fabsf(py_h);
    const float h0 = P.posy + static_cast<float>(P.top_index);
    Horizon z;
    z.a = K * c + py_t + eps * ma;
    z.b = K * d + py_h;
    z.eb = z.b + eps * mb <= 0.0f ? eps * mb : INFINITY;  // inf: the bound drops nothing
    z.scene = z.a <= 0.0f ? z.b * h0 + z.eb * fabsf(h0) : INFINITY;
    return z;
}

// Whether the cell may draw: it has runs and the topmost is not below the
// horizon for good.
__device__ __forceinline__ bool cell_alive(const RayParams& P, const Horizon& z, const Cell& c, float far) {
    const float h = P.posy + static_cast<float>(static_cast<int>((c.ey >> 16) & 1023u) << c.mip);
    const float bound = __fmaf_rn(z.a, z.a < 0.0f ? c.near : far, __fmaf_rn(z.b, h, z.eb * fabsf(h)));
    return (c.ey & 0xffffu) != 0u && !(bound < 0.0f);
}

// Casts ray x of frame P with one warp (lane k), using mask_words (S/32 words
// of shared memory) as its bitmask, in chunks of 32 DDA steps, lane k taking
// step k of each.
template <bool kCount, bool kHits>
__device__ __forceinline__ void cast_ray(const RayParams& P, int x, bool active, uint32_t* mask_words, uint32_t* recs,
                                         uint4* spans, uint32_t* list, int k, Counts& cnt) {
    const int S = P.S;
    const int words = (S + 31) >> 5;
    Mask mask{mask_words};

    uint32_t* my_recs = recs + threadIdx.x;
    const uint32_t* warp_recs = recs + (threadIdx.x & ~31u);
    SpanQueue q{spans, 0};
    Ray R;
    Walk W;
    bool live = false;
    if (active) {
        for (int w = k; w < words; w += kLanes) mask.w[w] = 0;
        live = setup_ray(P, x, R, W.d);
    } else {
        R.ymin = 0;
        R.ymax = -1;
    }
    __syncwarp();
    uint32_t* row = active ? P.raybuf + static_cast<size_t>(x) * S : nullptr;
    float* drow = active ? P.raydepth + static_cast<size_t>(x) * S : nullptr;
    rle_hit* hrow = nullptr;
    if constexpr (kHits) hrow = (active && P.rayhit) ? P.rayhit + static_cast<size_t>(x) * S : nullptr;
    const int ymin0 = R.ymin, ymax0 = R.ymax;

    if (live) {
        int ymin = R.ymin, ymax = R.ymax;
        W.mip = 0;
        W.z = 0;
        W.dz = 1;
        W.mapswitch = P.mapswitch0;
        W.zswitch = static_cast<float>(W.mapswitch);
        {
            // first step's switch test, the only one the camera height can
            // trigger: y_map_switch starts at position.y and only halves
            float y_map_switch = P.posy;
            while (W.z > W.zswitch || y_map_switch > 512.0f) {
                y_map_switch = y_map_switch * 0.5f;
                if (W.mip < P.nummaps - 1) W.mip++;
                W.d.g0x *= 2; W.d.g0y *= 2; W.d.g1x *= 2; W.d.g1y *= 2;
                W.d.gd0 *= 2; W.d.gd1 *= 2;
                W.mapswitch *= 2;
                W.zswitch = static_cast<float>(W.mapswitch);
                W.dz *= 2;
            }
        }
        W.cached = false;
        W.room = W.z > W.zswitch ? 0 : steps_unchecked(P, W);
        ChunkStep st;
        int nvalid = dda_chunk(P, W, k, st);
        Cell c = cell_of_step(P, R, k < nvalid, st);
        Horizon hz = horizon_bound(P, R, ymin);
        for (;;) {
            if (nvalid == 0) break;
            const bool ended = nvalid < kLanes;
            // ---- 1. this chunk's table entries, and under their latency the
            // next chunk's DDA steps ----
            const uint2 entry = cell_entry(P, c);
            int nvalid_next = 0;
            Cell c_next;
            c_next.near = 0.0f;
            if (!ended) {
                nvalid_next = dda_chunk(P, W, k, st);
                c_next = cell_of_step(P, R, k < nvalid_next, st);
            }
            c.ex = entry.x;
            c.ey = entry.y;
            // a cell ends where the next one begins
            const float far = __shfl_sync(kWarp, k == 0 ? c_next.near : c.near, (k + 1) % kLanes);

            if constexpr (kCount) {
                // with counters every valid cell goes through the exact walk
                const Edge edge = cell_edge(P, R, c.near, far);
                unsigned todo = __ballot_sync(kWarp, k < nvalid);
                // the reference ends the ray when its horizon closes, checked
                // at every step before the cell (:370)
                for (; todo && ymin < ymax; todo &= todo - 1) {
                    const int src = __ffs(todo) - 1;
                    cnt.cells++;
                    merge_cell<true>(P, R, mask, k, row, drow, hrow, cell_of(c, src),
                                        edge_of(edge, src), ymin, ymax, cnt);
                }
            } else {
                const bool alive = cell_alive(P, hz, c, far);
                if (__ballot_sync(kWarp, alive)) {
                    const Edge edge = cell_edge(P, R, c.near, far);
                    const int before = ymin;
                    int nrec = 0;
                    if (alive) nrec = scan_runs(P, R, mask, ymin, ymax, c, edge, my_recs, blockDim.x);
                    // ---- 3. the recorded runs, in the order of the walk ----
                    merge_chunk(P, R, mask, k, row, drow, hrow, c, edge, nrec, warp_recs, blockDim.x, list,
                                   ymin, ymax, q, cnt);
                    if (ymin != before) hz = horizon_bound(P, R, ymin);
                }
            }
            if (ymin >= ymax || ended) break;
            // Nothing further along this ray can be drawn once every run of
            // every later cell projects below the floating horizon (the
            // reference walks on to z_far without drawing).  Exact counters
            // need the full walk, so they keep it.
            if (!kCount) {
                const float t_end = __shfl_sync(kWarp, far, kLanes - 1);
                if (__fmaf_rn(hz.a, t_end, hz.scene) < 0.0f) break;
            }
            c = c_next;
            nvalid = nvalid_next;
        }
    }
    if (q.n > 0) flush_spans(P, R.pos3d_z_add, R.pos3d_y_add, q.e, q.n, k, row, drow, hrow);
    __syncwarp();

    // ---- coalesced fill of the samples no span coloured ----
    if (active) {
        for (int y = k; y < S; y += kLanes) {
            if (mask.get(y)) continue;
            const bool in = y >= ymin0 && y <= ymax0;
            row[y] = in ? kSky : 0u;
            drow[y] = in ? INFINITY : 0.0f;
            if (hrow) {
                rle_hit h = {0, 0, 0, 0, static_cast<uint8_t>(in ? 2 : 0)};
                hrow[y] = h;
            }
        }
    }
    __syncwarp();  // every lane has read the mask before the warp's next ray clears it
    if (kCount && active && k == 0) {
        // the lanes hold the same counts; lane 0 adds the ray's
        unsigned long long* c = reinterpret_cast<unsigned long long*>(P.counters);
        const unsigned long long v[6] = {cnt.cells, cnt.fetched, cnt.headers, cnt.runs, cnt.spans, cnt.pixels};
        for (int i = 0; i < 6; i++)
            if (v[i]) atomicAdd(&c[i], v[i]);
    }
    cnt = Counts();
}

// Shared memory of a raycast block: the warps' occupancy masks (`words` each,
// padded to 16 bytes), their span queues (one entry per lane), the merge's
// entry lists (one word per lane) and kRecs run records per thread.
__host__ __device__ constexpr int mask_region_words(int slots, int words) {
    return (slots * words + 3) & ~3;
}
__host__ __device__ constexpr size_t raycast_smem_bytes(int threads, int slots, int words) {
    return static_cast<size_t>(mask_region_words(slots, words)) * 4 +
           static_cast<size_t>(threads) * (kRecs * 3 * sizeof(uint32_t) + kQueueVecs * sizeof(uint4) + sizeof(uint32_t));
}
struct BlockSmem {
    int k, slots, slot;  // lane, warps of the block, this warp
    uint32_t* mask;      // this warp's mask
    uint32_t* recs;
    uint4* spans;        // this warp's queue
    uint32_t* list;      // this warp's list
    __device__ __forceinline__ BlockSmem(uint32_t* smem, int words) {
        k = threadIdx.x % kLanes;
        slots = blockDim.x / kLanes;
        slot = threadIdx.x / kLanes;
        mask = smem + slot * words;
        uint4* queues = reinterpret_cast<uint4*>(smem + mask_region_words(slots, words));
        spans = queues + slot * (kQueueVecs * kLanes);
        uint32_t* lists = reinterpret_cast<uint32_t*>(queues + blockDim.x * kQueueVecs);
        list = lists + slot * kLanes;
        recs = lists + blockDim.x;
    }
};

// One frame: ray slot s of block b casts ray b * slots + s.  kCount: the
// DETAIL_BENCH counters (exact walk of every cell); kHits: hit records.
template <bool kCount, bool kHits>
__global__ void __launch_bounds__(128, 4) raycast_kernel(const __grid_constant__ RayParams P) {
    extern __shared__ uint32_t smem[];
    const BlockSmem B(smem, (P.S + 31) >> 5);
    const int x = blockIdx.x * B.slots + B.slot;
    Counts cnt;
    // per-ray timing (rle_render_rays_timed): the first lane
    // stamps the ray's start and end; nothing else changes
    if (P.ray_time && B.k == 0 && x < P.rays) {
        rle_ray_time* t = P.ray_time + x;
        t->start_ns = global_ns();
        t->start_clock = static_cast<uint64_t>(clock64());
    }
    cast_ray<kCount, kHits>(P, x, x < P.rays, B.mask, B.recs, B.spans, B.list, B.k, cnt);
    if (P.ray_time && B.k == 0 && x < P.rays) {
        rle_ray_time* t = P.ray_time + x;
        t->end_clock = static_cast<uint64_t>(clock64());
        t->end_ns = global_ns();
        t->sm = sm_id();
        t->reserved = 0;
    }
}

// Many frames in one persistent launch.  The rays of all frames form one
// index space (ray_start[f] = first global ray of frame f); each warp takes
// `tile` consecutive rays at a time from a global counter until none are
// left, so long and short rays of every frame balance across the GPU.
template <bool kHits>
__global__ void __launch_bounds__(128, 4) raycast_batch_kernel(BatchHeader* hdr, const int* __restrict__ ray_start,
                                                               const RayParams* __restrict__ frames, int tile,
                                                               int max_words) {
    extern __shared__ uint32_t smem[];
    const BlockSmem B(smem, max_words);
    const int nframes = hdr->nframes;
    const int total = ray_start[nframes];
    Counts cnt;
    int f = 0;  // frame of the current ray (rays are taken in increasing order)
    // Guided self-scheduling: a warp claims up to `tile` adjacent rays, but
    // never more than half its fair share of what is left, so the last rays
    // go out one at a time and no warp is left with a long private tail.
    const int grab = tile;
    const int warps = static_cast<int>(gridDim.x) * B.slots;
    for (;;) {
        unsigned int t0 = 0, n = 1;
        if (B.k == 0) {
            const int seen = static_cast<int>(*reinterpret_cast<volatile unsigned int*>(&hdr->next_ray));
            n = static_cast<unsigned int>(max(1, min(grab, (total - seen) / (2 * warps))));
            t0 = atomicAdd(&hdr->next_ray, n);
        }
        t0 = __shfl_sync(kWarp, t0, 0);
        n = __shfl_sync(kWarp, n, 0);
        if (static_cast<int>(t0) >= total) break;
        const int t1 = min(static_cast<int>(t0) + static_cast<int>(n), total);
        for (int r = static_cast<int>(t0); r < t1; r++) {
            if (r < ray_start[f] || r >= ray_start[f + 1]) {
                int lo = 0, hi = nframes - 1;  // last frame with ray_start <= r
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (ray_start[mid] <= r) lo = mid;
                    else hi = mid - 1;
                }
                f = lo;
            }
            cast_ray<false, kHits>(frames[f], r - ray_start[f], true, B.mask, B.recs, B.spans, B.list, B.k, cnt);
        }
    }
}

// The largest launch (blocks of 128, ray maps of 16384 samples) has what a kernel
// may have without asking.  The limit that cudaFuncSetAttribute moves is the
// kernel's, in every thread and batch: moved to one launch's size, it refuses
// another's larger block.
static_assert(raycast_smem_bytes(128, 128 / kLanes, 16384 / 32) <= 48 * 1024, "dynamic shared memory of a launch");

template <bool kCount, bool kHits>
rle_status launch_variant(const RayParams& p, int threads, cudaStream_t stream) {
    const int words = (p.S + 31) >> 5;
    const int rays_per_block = threads / kLanes;
    const size_t smem = raycast_smem_bytes(threads, rays_per_block, words);
    const int blocks = (p.rays + rays_per_block - 1) / rays_per_block;
    forget_last_error();
    raycast_kernel<kCount, kHits><<<blocks, threads, smem, stream>>>(p);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("raycast launch: %s", cudaGetErrorString(e));
        return RLE_ERR_CUDA;
    }
    return RLE_OK;
}

rle_status launch_shape(const RayParams& p, int threads, cudaStream_t stream) {
    if (p.counters)
        return p.rayhit ? launch_variant<true, true>(p, threads, stream) : launch_variant<true, false>(p, threads, stream);
    return p.rayhit ? launch_variant<false, true>(p, threads, stream) : launch_variant<false, false>(p, threads, stream);
}

size_t batch_smem(int threads, int max_samples) {
    return raycast_smem_bytes(threads, threads / kLanes, (max_samples + 31) >> 5);
}

template <bool kHits>
rle_status batch_blocks(int threads, int max_samples, int* blocks) {
    const size_t smem = batch_smem(threads, max_samples);
    int dev = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, raycast_batch_kernel<kHits>,
                                                          threads, smem);
    if (e != cudaSuccess) {
        set_error("batch launch set-up: %s", cudaGetErrorString(e));
        return RLE_ERR_CUDA;
    }
    *blocks = sms * (per_sm > 0 ? per_sm : 1);
    return RLE_OK;
}

template <bool kHits>
rle_status batch_launch(const BatchRaycast& b, cudaStream_t stream) {
    const size_t smem = batch_smem(b.threads, b.max_samples);
    int blocks = b.blocks;
    if (blocks <= 0) {
        const rle_status st = batch_blocks<kHits>(b.threads, b.max_samples, &blocks);
        if (st != RLE_OK) return st;
    }
    forget_last_error();
    raycast_batch_kernel<kHits><<<blocks, b.threads, smem, stream>>>(
        b.header, b.ray_start, b.frames, b.tile, (b.max_samples + 31) >> 5);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("batch raycast launch: %s", cudaGetErrorString(e));
        return RLE_ERR_CUDA;
    }
    return RLE_OK;
}

}  // namespace

rle_status batch_grid_blocks(int threads, int max_samples, bool hits, int* blocks) {
    return hits ? batch_blocks<true>(threads, max_samples, blocks) : batch_blocks<false>(threads, max_samples, blocks);
}

rle_status launch_raycast_batch(const BatchRaycast& b, void* stream) {
    if (b.threads % 32 != 0 || b.threads <= 0 || b.threads > 128 || b.tile < 1) {
        set_error("batch: threads per block a multiple of 32 up to 128, tile >= 1");
        return RLE_ERR_INVALID_ARG;
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    return b.hits ? batch_launch<true>(b, s) : batch_launch<false>(b, s);
}

bool bounds_render(unsigned* out4, bool clear) {
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

rle_status launch_raycast(const RayParams& p, void* stream) {
    if (p.rays <= 0) return RLE_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int threads = p.threads_per_block > 0 ? p.threads_per_block : 128;
    if (threads % 32 != 0 || threads > 128) {
        set_error("raycast: threads per block must be a multiple of 32, at most 128");
        return RLE_ERR_INVALID_ARG;
    }
    return launch_shape(p, threads, s);
}

}  // namespace rle
