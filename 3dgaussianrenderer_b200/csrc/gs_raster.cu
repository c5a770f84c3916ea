// Tile rasteriser (replaces rasterizeTilesKernel, core/gaussian_render.cu:679-775).
//
// One CTA per tile.  The tile's depth-sorted entries are staged in shared
// memory (centre, conic + opacity, colour) and the pixels blend them front to
// back in FP32 with the reference's arithmetic.
//
// Termination:
//  * GS_TERM_REFERENCE: every pixel evaluates every entry; after every 32nd
//    entry of the tile's list the CTA stops once no in-image pixel has
//    T > 0.02 (the reference's test at :745).  Batches of 32 entries,
//    double-buffered so the gather of the next batch overlaps the blending
//    of this one.  Bit-identical to the reference kernel.
//  * GS_TERM_TMIN: a pixel stops once its T < t_min; a warp whose pixels are
//    all done skips the rest (warp ballot), the CTA stops when every pixel
//    is done.  Each warp first tests 32 staged splats at a time against its
//    8x4 pixel block (one splat per lane) and blends only the survivors
//    (ballot compaction).  A splat survives when its cutoff ellipse, where
//    opacity * exp(-q/2) = kCullAlpha, touches the block; the contributions
//    skipped are each below kCullAlpha (2^-18), so a pixel needs more than a
//    thousand of them to move by 1/255.
//
// One launch covers the tiles of all views of a frame.
#include "gs_kernels.h"
#include "gs_tilesort.cuh"
#include "gs_f32x2.cuh"

#include <algorithm>

namespace gs {

struct RasterSmem {
    float2* xy;
    float4* con;  // (a, b, c, opacity)
    float4* col;
    float4* box;  // cutoff box (x0, x1, y0, y1), GS_TERM_TMIN only
};

__device__ __forceinline__ void blend(const float cx, const float cy, const float2 c, const float4 k, const float4 col,
                                      float& r, float& g, float& b, float& T)
{
    const float dx = cx - c.x, dy = cy - c.y;
    const float q = k.x * dx * dx + k.z * dy * dy + 2.0f * k.y * dx * dy;
    const float density = __expf(-0.5f * q);
    const float alpha = k.w * __saturatef(density);
    r += col.x * T * alpha;
    g += col.y * T * alpha;
    b += col.z * T * alpha;
    T *= (1.0f - alpha);
}

__device__ __forceinline__ void cp_async(void* dst, const void* src, const int bytes_is_16)
{
    if (bytes_is_16)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Copies entry `s` (centre, conic, colour) into shared-memory slot `slot`.
__device__ __forceinline__ void stage_entry(const RasterArgs& a, const int s, const struct RasterSmem& sm,
                                            const int slot)
{
    cp_async(&sm.xy[slot], &a.xy[s], 0);
    cp_async(&sm.con[slot], &a.conic[s], 1);
    cp_async(&sm.col[slot], &a.color[s], 1);
}

// GS_TERM_TMIN from the reference's buffers (the stage API).
template <int TW, int TH>
__device__ __forceinline__ void raster_tile(const RasterArgs& a, const ViewParams& v, const int64_t gtile,
                                            const int local_tile, const RasterSmem& sm)
{
    constexpr int NT = TW * TH;
    constexpr int WX = TW / 8;  // warps per tile row
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int first = __ldg(&a.ranges[2 * gtile]);
    const int last = __ldg(&a.ranges[2 * gtile + 1]);
    const int count = last - first;
    const int tx = local_tile % v.tiles_x, ty = local_tile / v.tiles_x;
    const int wx0 = tx * TW + (warp % WX) * 8, wy0 = ty * TH + (warp / WX) * 4;
    const int px = wx0 + (lane & 7);
    const int py = wy0 + (lane >> 3);
    const bool inimg = px < v.width && py < v.height;
    if (count <= 0) {
        // the reference clears the image and skips empty tiles (main.cpp:363);
        // writing zeros here instead saves the separate clear
        if (a.write_empty && inimg) v.out[(int64_t)py * v.width + px] = make_uchar4(0, 0, 0, 0);
        return;
    }
    // pixel corner sample, gaussian_render.cu:701-704
    const float cx = (float)px * v.texel_x - 1.0f;
    const float cy = (float)py * v.texel_y - 1.0f;
    // this warp's 8x4 block in clip space
    const float bx0 = (float)wx0 * v.texel_x - 1.0f, bx1 = (float)(wx0 + 7) * v.texel_x - 1.0f;
    const float by0 = (float)wy0 * v.texel_y - 1.0f, by1 = (float)(wy0 + 3) * v.texel_y - 1.0f;

    float r = 0.0f, g = 0.0f, b = 0.0f;
    float T = 1.0f;
    bool done = !inimg;

    for (int base = 0; base < count; base += NT) {
        const int nb = min(NT, count - base);
        __syncthreads();
        if ((int)threadIdx.x < nb) {
            const int s = __ldg(&a.values[first + base + threadIdx.x]);
            const float4 col = __ldg(&a.color[s]);
            const float4 con = __ldg(&a.conic[s]);
            const float2 c = __ldg(&a.xy[s]);
            sm.xy[threadIdx.x] = c;
            sm.con[threadIdx.x] = make_float4(con.x, con.y, con.z, col.w);
            sm.col[threadIdx.x] = col;
            {
                float4 box;
                const float det = con.x * con.z - con.y * con.y;
                if (!(col.w > kCullAlpha)) {
                    box = make_float4(1e30f, -1e30f, 1e30f, -1e30f);  // contributes nothing
                } else if (!(det > 0.0f) || !(con.x > 0.0f) || !(con.z > 0.0f)) {
                    box = make_float4(-1e30f, 1e30f, -1e30f, 1e30f);  // degenerate: never cull
                } else {
                    const float qc = 2.0f * logf(col.w / kCullAlpha);
                    const float ex = sqrtf(qc * con.z / det), ey = sqrtf(qc * con.x / det);
                    box = make_float4(c.x - ex, c.x + ex, c.y - ey, c.y + ey);
                }
                sm.box[threadIdx.x] = box;
            }
        }
        __syncthreads();
        {
            for (int c0 = 0; c0 < nb; c0 += 32) {
                if (__all_sync(kFull, done)) break;
                const int j = c0 + lane;
                bool keep = false;
                if (j < nb) {
                    const float4 bx = sm.box[j];
                    keep = bx.x <= bx1 && bx.y >= bx0 && bx.z <= by1 && bx.w >= by0;
                }
                unsigned m = __ballot_sync(kFull, keep);
                while (m) {
                    const int k = c0 + __ffs(m) - 1;
                    m &= m - 1;
                    if (!done) {
                        blend(cx, cy, sm.xy[k], sm.con[k], sm.col[k], r, g, b, T);
                        if (T < a.t_min) done = true;
                    }
                }
            }
            if (__syncthreads_count(!done) == 0) break;
        }
    }

    if (inimg) {
        uchar4 qc;
        qc.x = r * 255;
        qc.y = g * 255;
        qc.z = b * 255;
        qc.w = 255;
        v.out[(int64_t)py * v.width + px] = qc;
    }
}

__device__ __forceinline__ void store_pixel(const ViewParams& v, const int px, const int py, const float r,
                                            const float g, const float b)
{
    uchar4 qc;
    qc.x = r * 255;
    qc.y = g * 255;
    qc.z = b * 255;
    qc.w = 255;
    v.out[(int64_t)py * v.width + px] = qc;
}

// ---- per-tile sort inside the raster CTA ----------------------------------------
//
// In tile-bucket frames a tile of at most fused_cap keys arrives unsorted;
// its CTA orders it in shared memory (gs_tilesort.cuh) before blending and
// reads the slots from there.  Larger tiles were sorted ahead of the raster
// and are read from `values`.

// Sorts a tile of up to CAP keys with the CTA's NT threads (CAP / NT keys
// per thread).  Returns the tile's sorted keys (sm.k), or null when the order
// is in a.values.  Every thread of the CTA must call it; where it sorts, it
// ends with a barrier.
template <int NT, int CAP>
__device__ __forceinline__ const uint64_t* fused_sort(const RasterArgs& a, const int first, const int count,
                                                      const tilesort::Smem& sm)
{
    if (!a.keys || count > a.fused_cap) return nullptr;
    if (count == 1) {
        if (threadIdx.x == 0) sm.k[0] = a.keys[first];
        __syncthreads();
        return sm.k;
    }
    const uint64_t* src = a.keys + first;
    if (count <= NT)
        tilesort::sort_tile<NT, 1>(src, count, a.slot_gi, sm, a.sort_prefix_bits);
    else if (count <= 2 * NT)
        tilesort::sort_tile<NT, 2>(src, count, a.slot_gi, sm, a.sort_prefix_bits);
    else if (count <= 4 * NT)
        tilesort::sort_tile<NT, 4>(src, count, a.slot_gi, sm, a.sort_prefix_bits);
    else if (CAP == 8 * NT || count <= 8 * NT)
        tilesort::sort_tile<NT, 8>(src, count, a.slot_gi, sm, a.sort_prefix_bits);
    else
        tilesort::sort_tile<NT, CAP / NT>(src, count, a.slot_gi, sm, a.sort_prefix_bits);
    return sm.k;
}

// Slot of the idx-th entry of the tile whose list starts at `first`.
__device__ __forceinline__ int slot_at(const RasterArgs& a, const uint64_t* sk, const int first, const int idx)
{
    return sk ? (int)(uint32_t)sk[idx] : __ldg(&a.values[first + idx]);
}

// The raster's times: its first CTA stamps the start.  The end is stamped by
// every warp of the last CTAs and of each tile of kStampKeys entries or more
// (the last writer stays): a tile that is drawn early, but is long, may end
// after all others.  A shorter one among the earlier CTAs takes 10 us or so, by
// which the end may be early at the most.  Stamps of all tiles would cost a
// frame whose images stream to the host 0.4 ms (24 views), and a short tile a
// good part of its own time.  Persistent CTAs end in any order: all of them stamp.
constexpr int kStampKeys = 512;
__device__ __forceinline__ void stamp_start(const RasterArgs& a)
{
    if (a.result && a.stamp_start && blockIdx.x == 0 && threadIdx.x == 0) stamp(a.result, kTimeRaster);
}
__device__ __forceinline__ void stamp_end(const RasterArgs& a, const int count)
{
    if (!a.result || !a.end_ctas || (threadIdx.x & 31) != 0) return;
    if (count >= kStampKeys || blockIdx.x + (unsigned)a.end_ctas >= gridDim.x) stamp(a.result, kTimeEnd);
}

// The view a global tile belongs to: binary search over the views' first tiles.
__device__ __forceinline__ const ViewParams& view_of_tile(const RasterArgs& a, const int64_t gtile)
{
    if (a.num_views <= 1) return a.view0;
    int vi = 0, hi = a.num_views - 1;
    while (vi < hi) {
        const int mid = (vi + hi + 1) >> 1;
        if (a.views[mid].tile_offset <= gtile)
            vi = mid;
        else
            hi = mid - 1;
    }
    return a.views[vi];
}

// ---- GS_TERM_REFERENCE ------------------------------------------------------------
//
// The reference's blend and termination, bit for bit: every pixel evaluates
// every entry, in batches of 32, and after each batch the tile stops once no
// pixel has T > 0.02.  The reference's expression
// (gaussian_render.cu:727-737) as nvcc contracts it:
//   q     = fma((2 b) dx, dy, fma(a dx, dx, (c dy) dy))
//   alpha = opacity * sat(exp(-0.5 q))
//   rgb   = fma(rgb_s T, alpha, rgb);   T = T (1 - alpha)
// Each lane owns NC columns x 2 rows of pixels, the rows of a column as one
// packed f32x2 pair, so an entry's shared-memory reads (40 bytes, broadcast),
// its row terms (dy, (c dy) dy) and its column terms (dx, a dx, 2 b dx) are
// shared by the lane's pixels.
// The FP32 pipe bounds the loop (73 % busy on the frame below): 13 packed operations (two cycles each) and 6
// scalar ones per entry and column pair.  On the 3M-Gaussian 1024x1024 frame
// the raster takes 0.42 ms, against 0.55 ms with two pixels per lane in scalar
// arithmetic (0.46 packed; 0.45 with four rows of one column per lane).
// The batches are double-buffered: the first warp starts asynchronous
// copies (cp.async, global -> shared, no registers held) of batch k + 1 and
// loads the indices of batch k + 2 before the tile blends batch k; the
// barrier that ends batch k publishes batch k + 1.
struct RefSmem {
    float2 xy[64];
    float4 con[64];  // (a, b, c, -)
    float4 col[64];  // (red, green, blue, opacity)
    int wild[2];     // the batch holds an entry whose exponent may be NaN
};

// Pixel layout of a tile: 8 lanes across, so a warp covers 8 NC x 8 pixels
// (a lane's two rows are 4 apart).
template <int TW, int TH, int COLS>
struct RefShape {
    static constexpr int NC = COLS;
    static constexpr int WX = TW / (8 * NC);  // warps across a tile
    static constexpr int NT = TW * TH / (2 * NC);
    static constexpr int CAP = TW * TH / 2 * kFusedIpt;
};

__device__ __forceinline__ float ex2_approx(const float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// exp(-q/2) = 2^p with p = -(log2(e) / 2) q, one product and one ex2.  The
// product and the constant leave p off by at most |p| (2^-24 + 2^-26) and ex2 is
// good to 2^-22 of its value, so the density is within 2^-22 + 3.8e-8 |q| of
// itself; a result below 2^-126, which changes no colour, is flushed to 0.
// gs_probe_density evaluates this form beside the call of __expf that the
// reference makes: on 16M values of q all results of 2^-126 and above are the
// same bits.
constexpr float kExponentOfQ = -0.72134752f;

// sat(2^p): clamped to 1 above and with NaN as 0.  Where p cannot be NaN (WILD
// false) the clamp is taken on p instead, which moves it from the FP32 pipe,
// the loop's bound, to the ALU: 2^0 is exactly 1 and 2^p is at most 1 for
// p <= 0.
template <bool WILD>
__device__ __forceinline__ float density_of(const float p)
{
    return WILD ? __saturatef(ex2_approx(p)) : ex2_approx(fminf(p, 0.0f));
}

// One entry into the lane's pixels.
template <int NC, bool WILD>
__device__ __forceinline__ void blend_ref(const float (&cx)[NC], const f2 cy, const RefSmem& sm, const int j,
                                          f2 (&R)[NC], f2 (&G)[NC], f2 (&B)[NC], f2 (&T)[NC])
{
    const float2 c = sm.xy[j];
    const float4 k = sm.con[j];
    const float4 col = sm.col[j];
    const f2 r2 = f2_dup(col.x), g2 = f2_dup(col.y), b2 = f2_dup(col.z), op2 = f2_dup(col.w);
    const f2 dy = f2_sub(cy, f2_dup(c.y));
    const f2 cdy2 = f2_mul(f2_mul(f2_dup(k.z), dy), dy);
    const float kb2 = 2.0f * k.y;
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        const float dx = __fsub_rn(cx[i], c.x);
        const f2 inner = f2_fma(f2_dup(__fmul_rn(k.x, dx)), f2_dup(dx), cdy2);
        const f2 p = f2_mul(f2_fma(f2_dup(__fmul_rn(kb2, dx)), dy, inner), f2_dup(kExponentOfQ));
        float p0, p1;
        f2_unpack(p, p0, p1);
        const f2 alpha = f2_mul(op2, f2_pack(density_of<WILD>(p0), density_of<WILD>(p1)));
        R[i] = f2_fma(f2_mul(r2, T[i]), alpha, R[i]);
        G[i] = f2_fma(f2_mul(g2, T[i]), alpha, G[i]);
        B[i] = f2_fma(f2_mul(b2, T[i]), alpha, B[i]);
        T[i] = f2_mul(T[i], f2_sub(f2_dup(1.0f), alpha));
    }
}

// Whether entry j's exponent might be NaN somewhere on the image: anything but
// a moderate centre and a conic whose products stay finite.
__device__ __forceinline__ bool wild_entry(const RefSmem& sm, const int j)
{
    const float2 c = sm.xy[j];
    const float4 k = sm.con[j];
    return !(fabsf(c.x) < 1e3f && fabsf(c.y) < 1e3f && fabsf(k.x) < 1e30f && fabsf(k.y) < 1e30f &&
             fabsf(k.z) < 1e30f);
}

// One tile; returns its entries.
template <int TW, int TH, int COLS>
__device__ __forceinline__ int raster_ref_tile(const RasterArgs& a, const ViewParams& v, const int64_t gtile,
                                               const int local_tile, RefSmem& sm,
                                               const tilesort::Smem& ts)
{
    using S = RefShape<TW, TH, COLS>;
    constexpr int NC = S::NC;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int first = a.ranges[2 * gtile];
    const int last = a.ranges[2 * gtile + 1];
    const int count = last - first;
    const int tx = local_tile % v.tiles_x, ty = local_tile / v.tiles_x;
    const int px = tx * TW + (warp % S::WX) * 8 * NC + (lane & 7) * NC;
    const int py0 = ty * TH + (warp / S::WX) * 8 + (lane >> 3), py1 = py0 + 4;
    const bool iny0 = py0 < v.height, iny1 = py1 < v.height;
    if (count <= 0) {
        // the reference clears the image and skips empty tiles (main.cpp:363);
        // writing zeros here instead saves the separate clear
        if (a.write_empty) {
#pragma unroll
            for (int i = 0; i < NC; ++i) {
                if (px + i >= v.width) continue;
                if (iny0) v.out[(int64_t)py0 * v.width + px + i] = make_uchar4(0, 0, 0, 0);
                if (iny1) v.out[(int64_t)py1 * v.width + px + i] = make_uchar4(0, 0, 0, 0);
            }
        }
        return 0;
    }
    const uint64_t* sk = fused_sort<S::NT, S::CAP>(a, first, count, ts);
    // pixel corner sample, gaussian_render.cu:701-704
    const f2 cy = f2_pack((float)py0 * v.texel_y - 1.0f, (float)py1 * v.texel_y - 1.0f);
    float cx[NC];
    f2 R[NC], G[NC], B[NC], T[NC];
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        cx[i] = (float)(px + i) * v.texel_x - 1.0f;
        R[i] = G[i] = B[i] = f2_dup(0.0f);
        T[i] = f2_dup(1.0f);
    }
    const RasterSmem rs = {sm.xy, sm.con, sm.col, nullptr};
    const bool loader = threadIdx.x < 32;
    const int t = (int)threadIdx.x;
    // the loader warp's copies have landed: flags the batch in slots [j0, j0 + 32)
    auto flag_wild = [&](const int j0, const int n) {
        const bool w = __any_sync(kFull, t < n && wild_entry(sm, j0 + t));
        if (t == 0) sm.wild[j0 >> 5] = w;
    };
    if (loader && t < count) stage_entry(a, slot_at(a, sk, first, t), rs, t);
    cp_async_commit();
    int idx_next = (loader && 32 + t < count) ? slot_at(a, sk, first, 32 + t) : 0;
    cp_async_wait_all();
    if (loader) flag_wild(0, count);
    __syncthreads();
    for (int base = 0; base < count; base += 32) {
        const int buf = (base >> 5) & 1;
        const int nb = min(32, count - base);
        const bool more = loader && base + 32 + t < count;
        if (more) stage_entry(a, idx_next, rs, 32 * (buf ^ 1) + t);
        cp_async_commit();
        const int n2 = base + 64 + t;
        const int idx2 = (loader && n2 < count) ? slot_at(a, sk, first, n2) : 0;
        const int j0 = 32 * buf;
        if (sm.wild[buf]) {
            for (int j = j0; j < j0 + nb; ++j) blend_ref<NC, true>(cx, cy, sm, j, R, G, B, T);
        } else if (nb == 32) {
#pragma unroll 8
            for (int j = j0; j < j0 + 32; ++j) blend_ref<NC, false>(cx, cy, sm, j, R, G, B, T);
        } else {
            for (int j = j0; j < j0 + nb; ++j) blend_ref<NC, false>(cx, cy, sm, j, R, G, B, T);
        }
        idx_next = idx2;
        cp_async_wait_all();
        if (loader && base + 32 < count) flag_wild(32 * (buf ^ 1), count - base - 32);
        bool open = false;
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            float t0, t1;
            f2_unpack(T[i], t0, t1);
            open |= px + i < v.width && ((iny0 && t0 > 0.02f) || (iny1 && t1 > 0.02f));
        }
        if (!__syncthreads_or(open)) break;
    }
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        if (px + i >= v.width) continue;
        float r0, r1, g0, g1, b0, b1;
        f2_unpack(R[i], r0, r1);
        f2_unpack(G[i], g0, g1);
        f2_unpack(B[i], b0, b1);
        if (iny0) store_pixel(v, px + i, py0, r0, g0, b0);
        if (iny1) store_pixel(v, px + i, py1, r1, g1, b1);
    }
    return count;
}

// One CTA per tile of every view, in the raster order when there is one.
// 640 threads per SM (96 registers, at which the wide lanes spill 76 bytes a
// thread, 228 in 16x8 tiles): the FP32 pipe is busy with 20 warps, and more of
// them only slow the heaviest tiles down (768 threads: raster +3 %).
template <int TW, int TH, int COLS>
__global__ void __launch_bounds__(RefShape<TW, TH, COLS>::NT, 640 / RefShape<TW, TH, COLS>::NT) raster_ref_kernel(RasterArgs a)
{
    using S = RefShape<TW, TH, COLS>;
    __shared__ RefSmem sm;
    __shared__ uint64_t s_k[S::CAP];
    __shared__ int32_t s_v[S::CAP];
    __shared__ int32_t s_bexcl[256], s_dcount[256], s_scan[S::NT / 32];
    __shared__ uint64_t s_red[2 * (S::NT / 32)];
    tilesort::Smem ts;
    ts.k = s_k;
    ts.v = s_v;
    ts.whist = reinterpret_cast<uint32_t*>(s_k);
    ts.bexcl = s_bexcl;
    ts.dcount = s_dcount;
    ts.scan = s_scan;
    ts.red = s_red;
    ts.run = nullptr;
    if (a.overlap) frame_step_begin();
    const int64_t gtile = a.order ? (int64_t)a.order[a.tile_base + blockIdx.x] : a.tile_base + blockIdx.x;
    const ViewParams& v = view_of_tile(a, gtile);
    stamp_start(a);
    stamp_end(a, raster_ref_tile<TW, TH, COLS>(a, v, gtile, (int)(gtile - v.tile_offset), sm, ts));
}

template <int TW, int TH>
__global__ void __launch_bounds__(TW * TH, 2048 / (TW * TH) * 5 / 8) raster_kernel(RasterArgs a)
{
    __shared__ float2 s_xy[TW * TH];
    __shared__ float4 s_con[TW * TH];
    __shared__ float4 s_col[TW * TH];
    __shared__ float4 s_box[TW * TH];
    const RasterSmem sm = {s_xy, s_con, s_col, s_box};
    raster_tile<TW, TH>(a, a.view0, (int64_t)blockIdx.x + a.view0.tile_offset, (int)blockIdx.x, sm);
}

// ---- GS_TERM_TMIN from raster records --------------------------------------
//
// The frame pipeline's kernel for the T_min mode.  One CTA per tile (all
// views' tiles in one grid), no CTA-wide barrier after the tile's sort: each
// warp owns BPW 8x8 pixel blocks side by side (2, or 1 where a tile is one
// block), 32 / BPW lanes to a block, and walks the tile's sorted list on its
// own, 32 entries at a time -- a lane tests the cull extents of one entry's
// record (48 bytes, gathered through L1, shared by the tile's warps) against
// the blocks; each block's survivors are copied in list order into its own
// shared-memory slots (rank = popcount of the ballot below the lane) and the
// block's lanes blend them into their pixels, BPW columns x 2 rows each.  The
// two halves of a warp walk their blocks' slots side by side; the shorter
// list is filled up with entries of weight zero (7 % more evaluations on a
// 1080p view of 1M Gaussians).
// Blend per pixel: alpha = 2^(A dx^2 + B dx dy + C dy^2 + L) (opacity
// folded in as L = log2(opacity); the conics are positive definite, so
// alpha <= opacity), w = T alpha, colour += rgb w, T -= w, in packed f32x2
// pairs of a column's two rows.  A block stops after the chunk in which all
// its pixels reached T < t_min; a pixel that got there earlier keeps blending
// until then, which adds less than t_min to its colour (the w that follow sum
// to less than its T).
//
// Every lane of a block reads every survivor of it.  With one block per warp
// and two pixels per lane those reads took 9 cycles of the SM's shared-memory
// path per 64 evaluations and bound the loop; two blocks per warp, four
// pixels per lane, halve them, share the row term (dy) and the column terms
// (A dx^2 + L, B dx) among the pixels.  What is left is spread: on four views of
// 3M Gaussians the issue slots are 67 % busy, the shared-memory path 66 %, the
// FP32 pipe 63 % (38 cycles per entry of a warp) and the ex2 unit 53 % (32
// cycles), and warps wait for one another's turn (not_selected, math_pipe_throttle).
// Raster of the 64-view batch of 3M Gaussians 14.7 -> 12.8 ms, of eight
// 1280x720 views of 1M 0.99 -> 0.83 ms, of one 1080p view 0.195 -> 0.175 ms.
// 640 threads per SM (96 registers, at which the wide lanes spill 88 bytes a
// thread, 132 in 16x8 tiles): 768 with 80 registers take 13.2 ms, 896 and 1024
// take 14.0 ms.
template <int TW, int TH, int BLOCKS>
struct RecShape {
    static constexpr int BPW = BLOCKS;              // 8x8 blocks per warp, side by side
    static constexpr int WX = TW / (8 * BPW);       // warps across a tile
    static constexpr int NT = TW * TH / (2 * BPW);  // threads: 2 BPW pixels each
    static constexpr int CAP = TW * TH / 2 * kFusedIpt;
    // CTAs per SM.  A tile of one block is a CTA of one warp: as many as an SM
    // takes (64 registers), since most such tiles are short and wait for memory
    // (8x8 tiles, eight views of 300k: 370 -> 333 us; sixteen of 3M unchanged).
    static constexpr int PER_SM = (TW * TH == 64 ? 1024 : 640) / NT;
};

// Shared memory of the record raster: the sort's buffers and, once the tile
// is sorted, in their place the tile's slots in blend order and every block's
// survivors, double-buffered.
constexpr int kRecStep = 32;  // entries a warp culls and stages at a time
template <int TW, int TH, int BLOCKS>
union RecSmem {
    using S = RecShape<TW, TH, BLOCKS>;
    static constexpr int NB = TW * TH / 64;
    struct {
        uint64_t k[S::CAP];
        int32_t v[S::CAP];
        int32_t bexcl[256];
        int32_t dcount[256];
        int32_t scan[S::NT / 32];
        uint64_t red[2 * (S::NT / 32)];
    } sort;
    struct {
        uint32_t order[S::CAP];
        float4 con[NB][2][kRecStep];  // (A, B, C, L)
        float4 col[NB][2][kRecStep];  // (red, green, blue, -)
        float2 xy[NB][2][kRecStep];
    } r;
};

// One tile of the record raster.  Every thread of the CTA must call it (the
// fused sort synchronises the CTA).  CHUNK (32 or 64) = the entries between
// two tests of whether a block is done.  Returns the tile's entries.
template <int TW, int TH, int CHUNK, int BLOCKS>
__device__ __forceinline__ int raster_rec_tile(const RasterArgs& a, const int64_t gtile, RecSmem<TW, TH, BLOCKS>& sm)
{
    using S = RecShape<TW, TH, BLOCKS>;
    constexpr int BPW = S::BPW;
    constexpr int LPB = 32 / BPW;  // lanes per block
    constexpr int LX = 8 / BPW;    // lanes across a block
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // the range's loads do not wait for the search of the view
    const int first = a.ranges[2 * gtile];
    const int count = a.ranges[2 * gtile + 1] - first;
    const ViewParams& v = view_of_tile(a, gtile);
    const int local_tile = (int)(gtile - v.tile_offset);
    const int tx = local_tile % v.tiles_x, ty = local_tile / v.tiles_x;
    // the warp's blocks: (wx0 + 8 b, wy0)
    const int wx0 = tx * TW + (warp % S::WX) * 8 * BPW, wy0 = ty * TH + (warp / S::WX) * 8;
    const int half = lane / LPB, sub = lane % LPB;
    const int px = wx0 + 8 * half + (sub % LX) * BPW, py0 = wy0 + sub / LX, py1 = py0 + 4;
    const bool iny0 = py0 < v.height, iny1 = py1 < v.height;
    if (count <= 0) {
        if (a.write_empty) {
#pragma unroll
            for (int c = 0; c < BPW; ++c) {
                if (px + c >= v.width) continue;
                if (iny0) v.out[(int64_t)py0 * v.width + px + c] = make_uchar4(0, 0, 0, 0);
                if (iny1) v.out[(int64_t)py1 * v.width + px + c] = make_uchar4(0, 0, 0, 0);
            }
        }
        return 0;
    }
    const bool sorted_here = a.keys && count <= a.fused_cap;
    if (sorted_here) {
        tilesort::Smem ts;
        ts.k = sm.sort.k;
        ts.v = sm.sort.v;
        ts.whist = reinterpret_cast<uint32_t*>(sm.sort.k);
        ts.bexcl = sm.sort.bexcl;
        ts.dcount = sm.sort.dcount;
        ts.scan = sm.sort.scan;
        ts.red = sm.sort.red;
        ts.run = nullptr;
        fused_sort<S::NT, S::CAP>(a, first, count, ts);
        // the keys give way to their slots
        uint32_t o[S::CAP / S::NT];
#pragma unroll
        for (int i = 0; i < S::CAP / S::NT; ++i) {
            const int p = i * S::NT + (int)threadIdx.x;
            if (p < count) o[i] = (uint32_t)sm.sort.k[p];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < S::CAP / S::NT; ++i) {
            const int p = i * S::NT + (int)threadIdx.x;
            if (p < count) sm.r.order[p] = o[i];
        }
        __syncthreads();
    }
    auto slot = [&](const int j) {
        return sorted_here ? (int)sm.r.order[j] : __ldg(&a.values[first + j]);
    };
    const f2 cy = f2_pack((float)py0 * v.texel_y - 1.0f, (float)py1 * v.texel_y - 1.0f);
    const float by0 = (float)wy0 * v.texel_y - 1.0f, by1 = (float)(wy0 + 7) * v.texel_y - 1.0f;
    float cx[BPW], bx0[BPW], bx1[BPW];
    f2 T[BPW], CR[BPW], CG[BPW], CB[BPW];
    bool out = true;
#pragma unroll
    for (int c = 0; c < BPW; ++c) {
        cx[c] = (float)(px + c) * v.texel_x - 1.0f;
        bx0[c] = (float)(wx0 + 8 * c) * v.texel_x - 1.0f;
        bx1[c] = (float)(wx0 + 8 * c + 7) * v.texel_x - 1.0f;
        // pixels outside the image start done (T = 0)
        const bool in0 = px + c < v.width && iny0, in1 = px + c < v.width && iny1;
        T[c] = f2_pack(in0 ? 1.0f : 0.0f, in1 ? 1.0f : 0.0f);
        CR[c] = CG[c] = CB[c] = f2_dup(0.0f);
        out = out && !in0 && !in1;
    }
    const float tmin = a.t_min;
    const unsigned lt = lanemask_lt();
    // block b is done when all its lanes are: bits [LPB b, LPB b + LPB)
    unsigned donemask = __ballot_sync(kFull, out);
    auto block_done = [&](const int b) {
        const unsigned m = BPW == 1 ? kFull : 0xFFFFu << (16 * b);
        return (donemask & m) == m;
    };
    const int blk = BPW * warp + half;  // this lane's block in the tile

    // Software pipeline over steps of 32 entries: while step i is blended, the
    // survivors of step i + 1 are on their way into the other buffer (cp.async),
    // the cull records of step i + 2 into registers and the slots of step
    // i + 3 are read.
    auto load_slot = [&](const int j) { return j < count ? slot(j) : -1; };
    auto load_cull = [&](const int s) { return s >= 0 ? __ldg(a.rec + 3 * (int64_t)s) : make_float4(0.f, 0.f, 0.f, 0.f); };
    int cnt[BPW];  // survivors of the step staged last
    auto stage = [&](const int s, const float4 q, const int buf) {
        const bool row = s >= 0 && (q.y - q.w <= by1) && (q.y + q.w >= by0);
#pragma unroll
        for (int b = 0; b < BPW; ++b) {
            const bool keep = row && !block_done(b) && (q.x - q.z <= bx1[b]) && (q.x + q.z >= bx0[b]);
            const unsigned bal = __ballot_sync(kFull, keep);
            if (keep) {
                const int o = BPW * warp + b, k = __popc(bal & lt);
                const float4* rp = a.rec + 3 * (int64_t)s;
                cp_async(&sm.r.con[o][buf][k], rp + 1, 1);
                cp_async(&sm.r.col[o][buf][k], rp + 2, 1);
                sm.r.xy[o][buf][k] = make_float2(q.x, q.y);
            }
            cnt[b] = __popc(bal);
        }
        cp_async_commit();
    };
    int s1 = load_slot(lane);
    int s2 = load_slot(32 + lane), s3 = load_slot(64 + lane);
    float4 q1 = load_cull(s1);
    stage(s1, q1, 0);
    q1 = load_cull(s2);
    for (int base = 0, buf = 0; base < count; base += kRecStep, buf ^= 1) {
        int now[BPW];
#pragma unroll
        for (int b = 0; b < BPW; ++b) now[b] = block_done(b) ? 0 : cnt[b];
        stage(s2, q1, buf ^ 1);
        s2 = s3;
        q1 = load_cull(s3);
        s3 = load_slot(base + 96 + lane);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        int n = now[0];
        if (BPW > 1) {
            __syncwarp();  // every lane's copies have landed: a done block's slots are overwritten
            // fill the shorter list up with entries that change nothing (2^-1e30 = 0)
            n = max(now[0], now[BPW - 1]);
            const int mine = half ? now[BPW - 1] : now[0];
            for (int k = mine + sub; k < n; k += LPB) {
                sm.r.con[blk][buf][k] = make_float4(0.f, 0.f, 0.f, -1e30f);
                sm.r.col[blk][buf][k] = make_float4(0.f, 0.f, 0.f, 0.f);
                sm.r.xy[blk][buf][k] = make_float2(0.f, 0.f);
            }
        }
        __syncwarp();  // this step's slots visible to the whole warp
#pragma unroll 4
        for (int k = 0; k < n; ++k) {
            const float2 c = sm.r.xy[blk][buf][k];
            const float4 e = sm.r.con[blk][buf][k];
            const float4 q = sm.r.col[blk][buf][k];
            const f2 dy = f2_sub(cy, f2_dup(c.y));
            const f2 C = f2_dup(e.z), red = f2_dup(q.x), green = f2_dup(q.y), blue = f2_dup(q.z);
#pragma unroll
            for (int i = 0; i < BPW; ++i) {
                const float dx = cx[i] - c.x;
                const f2 adx2 = f2_dup(fmaf(__fmul_rn(e.x, dx), dx, e.w));  // A dx^2 + L
                const f2 bdx = f2_dup(__fmul_rn(e.y, dx));
                float p0, p1;
                f2_unpack(f2_fma(f2_fma(C, dy, bdx), dy, adx2), p0, p1);
                const f2 w = f2_mul(T[i], f2_pack(ex2_approx(p0), ex2_approx(p1)));
                CR[i] = f2_fma(red, w, CR[i]);
                CG[i] = f2_fma(green, w, CG[i]);
                CB[i] = f2_fma(blue, w, CB[i]);
                T[i] = f2_sub(T[i], w);
            }
        }
        __syncwarp();  // this buffer is rewritten by the next step
        if (CHUNK == kRecStep || (base & kRecStep) || base + kRecStep >= count) {
            bool done = true;
#pragma unroll
            for (int c = 0; c < BPW; ++c) {
                float t0, t1;
                f2_unpack(T[c], t0, t1);
                done = done && t0 < tmin && t1 < tmin;
            }
            donemask = __ballot_sync(kFull, done);
        }
        if (donemask == kFull) break;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");  // none in flight when the CTA goes on or ends
#pragma unroll
    for (int c = 0; c < BPW; ++c) {
        if (px + c >= v.width) continue;
        float r0, r1, g0, g1, b0, b1;
        f2_unpack(CR[c], r0, r1);
        f2_unpack(CG[c], g0, g1);
        f2_unpack(CB[c], b0, b1);
        if (iny0) store_pixel(v, px + c, py0, r0, g0, b0);
        if (iny1) store_pixel(v, px + c, py1, r1, g1, b1);
    }
    return count;
}

// One CTA per tile of [tile_base, tile_base + grid), in the raster order.
template <int TW, int TH, int CHUNK, int BLOCKS>
__global__ void __launch_bounds__(RecShape<TW, TH, BLOCKS>::NT, RecShape<TW, TH, BLOCKS>::PER_SM) raster_rec_kernel(RasterArgs a)
{
    __shared__ __align__(16) unsigned char smem[sizeof(RecSmem<TW, TH, BLOCKS>)];
    RecSmem<TW, TH, BLOCKS>& sm = *reinterpret_cast<RecSmem<TW, TH, BLOCKS>*>(smem);
    if (a.overlap) frame_step_begin();
    const int64_t gtile = a.order ? (int64_t)a.order[a.tile_base + blockIdx.x] : a.tile_base + blockIdx.x;
    stamp_start(a);
    stamp_end(a, raster_rec_tile<TW, TH, CHUNK, BLOCKS>(a, gtile, sm));
}

// Persistent CTAs (as many as fit on the SMs at once) that pull tiles from
// an atomic queue over the raster order (heavy tiles first) until it runs
// dry.
template <int TW, int TH, int CHUNK, int BLOCKS>
__global__ void __launch_bounds__(RecShape<TW, TH, BLOCKS>::NT, RecShape<TW, TH, BLOCKS>::PER_SM)
    raster_rec_persistent_kernel(RasterArgs a)
{
    __shared__ __align__(16) unsigned char smem[sizeof(RecSmem<TW, TH, BLOCKS>)];
    RecSmem<TW, TH, BLOCKS>& sm = *reinterpret_cast<RecSmem<TW, TH, BLOCKS>*>(smem);
    __shared__ int64_t s_tile;
    if (a.overlap) frame_step_begin();
    stamp_start(a);
    for (;;) {
        if (threadIdx.x == 0) {
            const int64_t k = (int64_t)atomicAdd(a.tile_counter, 1ull);
            s_tile = k < a.num_tiles_total ? (a.order ? (int64_t)a.order[a.tile_base + k] : a.tile_base + k) : -1;
        }
        __syncthreads();
        const int64_t gtile = s_tile;
        if (gtile < 0) break;
        raster_rec_tile<TW, TH, CHUNK, BLOCKS>(a, gtile, sm);
        __syncthreads();  // s_tile and the sort's shared memory are reused
    }
    stamp_end(a, kStampKeys);
}

template <int TW, int TH, int CHUNK, int BLOCKS>
static void launch_rec(const RasterArgs& a, bool persistent, int num_sms, cudaStream_t st)
{
    if (a.num_tiles_total <= 0) return;
    if (!persistent) {
        launch_frame_step(raster_rec_kernel<TW, TH, CHUNK, BLOCKS>, (unsigned)a.num_tiles_total,
                          RecShape<TW, TH, BLOCKS>::NT, 0, st, a.overlap != 0, a);
        return;
    }
    static int per_sm = 0;  // same on every B200; queried once
    if (per_sm == 0) {
        int x = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&x, raster_rec_persistent_kernel<TW, TH, CHUNK, BLOCKS>,
                                                      RecShape<TW, TH, BLOCKS>::NT, 0);
        per_sm = std::max(x, 1);
    }
    const int64_t grid = std::min<int64_t>((int64_t)per_sm * num_sms, a.num_tiles_total);
    launch_frame_step(raster_rec_persistent_kernel<TW, TH, CHUNK, BLOCKS>, (unsigned)grid, RecShape<TW, TH, BLOCKS>::NT, 0, st,
                      a.overlap != 0, a);
}

// A launch of few tiles lasts as long as its longest ones, so it gives a tile
// twice the warps, of half the pixels each; many tiles are a matter of
// throughput, where the shared reads and terms of the wide lanes pay.  Raster,
// twice the warps against wide lanes: 300 tiles 8 / 12 us (reference mode 12 /
// 16), 1200 tiles 41 / 59 (88 / 116), 1900 tiles 38 / 49 (80 / 94), 2800 tiles
// 62 / 63 (84 / 93); 4096 tiles (397 / 368), 8160 tiles 172 / 153.
constexpr int kSmallTilesPerSm = 20;

template <int TW, int TH, int WIDE>
static void launch_width(const RasterArgs& a, int termination, int num_sms, cudaStream_t st)
{
    const unsigned tiles = (unsigned)a.num_tiles_total;
    if (termination == 0)
        launch_frame_step(raster_ref_kernel<TW, TH, WIDE>, tiles, RefShape<TW, TH, WIDE>::NT, 0, st, a.overlap != 0, a);
    else if (!a.rec)
        raster_kernel<TW, TH><<<tiles, TW * TH, 0, st>>>(a);
    else if (a.rec_chunk == 64)
        launch_rec<TW, TH, 64, WIDE>(a, a.rec_persistent != 0, num_sms, st);
    else
        launch_rec<TW, TH, 32, WIDE>(a, a.rec_persistent != 0, num_sms, st);
}

template <int TW, int TH>
static void launch_shape(const RasterArgs& a, int termination, int num_sms, cudaStream_t st)
{
    if (a.num_tiles_total <= 0) return;
    if (a.num_tiles_total <= (int64_t)kSmallTilesPerSm * num_sms)
        launch_width<TW, TH, 1>(a, termination, num_sms, st);
    else
        launch_width<TW, TH, TW / 8>(a, termination, num_sms, st);
}

// gs_probe_density: the reference raster's density, the form of batches that
// may hold a NaN and the other one, and the reference's expression.
__global__ void __launch_bounds__(256) density_probe_kernel(const int64_t n, const float* __restrict__ q,
                                                            float* __restrict__ wild, float* __restrict__ tame,
                                                            float* __restrict__ expf_form)
{
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    float p, unused;
    f2_unpack(f2_mul(f2_dup(q[i]), f2_dup(kExponentOfQ)), p, unused);
    wild[i] = density_of<true>(p);
    tame[i] = density_of<false>(p);
    expf_form[i] = __saturatef(__expf(__fmul_rn(-0.5f, q[i])));
}

void launch_density_probe(const int64_t n, const float* q, float* wild, float* tame, float* expf_form, cudaStream_t st)
{
    if (n <= 0) return;
    density_probe_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, q, wild, tame, expf_form);
}

void launch_raster(const RasterArgs& a, int tile_w, int tile_h, int termination, int num_sms, cudaStream_t st)
{
    if (tile_w == 16 && tile_h == 16)
        launch_shape<16, 16>(a, termination, num_sms, st);
    else if (tile_w == 16 && tile_h == 8)
        launch_shape<16, 8>(a, termination, num_sms, st);
    else
        launch_shape<8, 8>(a, termination, num_sms, st);
}

}  // namespace gs
