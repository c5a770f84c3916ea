// Tile-bucket ordering of the frame pipeline: the whole-frame replacement
// for the reference's buildTileList + sortTileList + evaluateTileRanges
// (core/gaussian_render.cu:312-677).
//
// The reference emits (tile << 32 | depth, index) keys, radix-sorts all of
// them on tile and depth bits, then finds each tile's range.  Here the frame
// kernel has already counted every tile's keys, so:
//   1. tile scan   -- exclusive scan of the tile counts = each tile's range;
//   2. bucket emit -- every overlap is written straight into its tile's
//                     range, at the rank its count gave it, as
//                     (depth << 32 | slot);
//   3. tile sort   -- each tile's keys are ordered by depth in shared
//                     memory (LSD radix over only the depth bits that vary
//                     inside the tile), equal depths by view * n + i; small
//                     tiles by the raster CTA right before it blends them,
//                     larger ones by a separate kernel.
// The result per tile is exactly the order of a stable sort of the
// reference's keys emitted in Gaussian order: depth first, index among equal
// depths.  Each key crosses HBM a few times (overlap list, emit, sort read)
// instead of twice per radix pass.
#include "gs_kernels.h"
#include "gs_tilesort.cuh"

#include <algorithm>

namespace gs {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

// Exclusive block scan of one int64 per thread; every thread must call it.
__device__ __forceinline__ int64_t excl_scan_block(const int64_t v, int64_t* s_tmp)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) s_tmp[warp] = incl;
    __syncthreads();
    int64_t prefix = 0;
    for (int w = 0; w < warp; ++w) prefix += s_tmp[w];
    __syncthreads();
    return prefix + incl - v;
}

}  // namespace

// Raster order: tiles go to the rasteriser by falling key count, in classes of
// half an octave (class 0 the heaviest), so that the longest CTAs start first
// and the last wave is made of the shortest.
//
// Tiles of fewer than 16 keys, the empty ones among them, are one class: with
// the empty tiles in a class of their own, at the end, a frame of many had a
// phase of nothing but CTA launches (raster of 17 views of 14k Gaussians in
// 384000 tiles of 8x8, half of them empty: 449 against 397 us).
__device__ __forceinline__ int order_class(const uint32_t count)
{
    if (count < 16) return kOrderClasses - 9;
    const int l = 31 - __clz((int)count);
    const int half = 2 * l + (l > 0 ? (int)((count >> (l - 1)) & 1u) : 0);
    return kOrderClasses - 2 - min(half, kOrderClasses - 2);
}

// The raster group of a tile.
__device__ __forceinline__ int group_of(const int64_t* group_tile, const int groups, const int64_t tile)
{
    int g = 0;
    while (g + 1 < groups && group_tile[g + 1] <= tile) ++g;
    return g;
}

// ---- 1. tile scan -------------------------------------------------------------

__global__ void __launch_bounds__(kThreads) tile_scan_kernel(const __grid_constant__ TileScanArgs a)
{
    constexpr int IPT = kTileScanItems / kThreads;
    __shared__ int64_t s_tmp[kWarps];
    __shared__ int64_t s_base;
    __shared__ int64_t s_blk;
    __shared__ unsigned int s_class[kMaxRasterGroups * kOrderClasses];
    const int classes = a.groups * kOrderClasses;
    for (int k = threadIdx.x; k < classes; k += kThreads) s_class[k] = 0u;
    frame_step_begin();
    if (threadIdx.x == 0) s_blk = (int64_t)atomicAdd(a.block_counter, 1ull);
    __syncthreads();
    const int64_t blk = s_blk;
    const int64_t nblk = (a.tiles + kTileScanItems - 1) / kTileScanItems;
    if (blk >= nblk) return;
    const uint32_t epoch = a.epoch_dev ? *a.epoch_dev : a.epoch;

    // thread t owns tiles [first, first + IPT) of this block
    const int64_t first = blk * kTileScanItems + (int64_t)threadIdx.x * IPT;
    uint32_t c[IPT];
    int64_t sum = 0;
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
        c[j] = first + j < a.tiles ? a.count[first + j] : 0u;
        sum += c[j];
    }
    // leave the counts zeroed for the next frame (saves a clear per frame)
#pragma unroll
    for (int j = 0; j < IPT; ++j)
        if (first + j < a.tiles) {
            if (c[j]) a.count[first + j] = 0u;
            atomicAdd(&s_class[order_class(c[j]) + kOrderClasses * group_of(a.group_tile, a.groups, first + j)], 1u);
        }
    const int64_t excl = excl_scan_block(sum, s_tmp);
    if (threadIdx.x == kThreads - 1) {
        const uint64_t agg = (uint64_t)(excl + sum);
        uint64_t prev = 0;
        uint64_t* st = a.status + blk;
        if (blk == 0) {
            store_status(st, status_word(kFlagP, epoch, agg));
        } else {
            store_status(st, status_word(kFlagA, epoch, agg));
            prev = look_back(a.status, blk, 1, epoch, a.err, kErrTimeout);
            store_status(st, status_word(kFlagP, epoch, prev + agg));
        }
        s_base = (int64_t)prev;
        if (blk == nblk - 1) {
            const int64_t total = (int64_t)(prev + agg);
            *a.total = total;
            *a.overflow = total > a.capacity || (int64_t)(*a.slot_counter >> 32) > a.chunk_capacity ||
                          (int64_t)*a.unit_count > a.unit_capacity;
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < classes; k += kThreads)
        if (s_class[k]) atomicAdd(&a.class_tiles[k], s_class[k]);
    int64_t run = s_base + excl;
    const int64_t cap = a.capacity;
#pragma unroll
    for (int j = 0; j < IPT; ++j) {
        const int64_t t = first + j;
        if (t < a.tiles) {
            if (c[j] > (uint32_t)kTileSortSmemKeys)
                a.big_list[a.tiles + atomicAdd(a.huge_count, 1u)] = (int32_t)t;
            else if (c[j] > (uint32_t)a.fused_cap)
                a.big_list[atomicAdd(a.big_count, 1u)] = (int32_t)t;
            const int64_t lo = run < cap ? run : cap;
            const int64_t hi = run + c[j] < cap ? run + c[j] : cap;
            a.ranges[2 * t] = (int32_t)lo;
            a.ranges[2 * t + 1] = (int32_t)hi;
        }
        run += c[j];
    }
}

void launch_tile_scan(const TileScanArgs& a, cudaStream_t st)
{
    const int64_t blocks = (a.tiles + kTileScanItems - 1) / kTileScanItems;
    if (blocks <= 0) return;
    launch_frame_step(tile_scan_kernel, (unsigned)blocks, kThreads, 0, st, a.overlap != 0, a);
}

// ---- 2. bucket emit -----------------------------------------------------------
//
// The raster order of the tiles first (their classes' sizes are the scan's),
// then one warp per chunk of the overlap list, four chunks in flight per warp.
// Each place reads its overlap (8 bytes), its slot's depth and its tile's start
// and writes one key; there is no chain longer than three loads.
// The blocks (as many as fit) take batches of chunks in order from a counter:
// a tile's next keys are then written close together in time and its sectors
// leave L2 full, where a fixed stride lets fast blocks run ahead and sectors
// are fetched and written back twice (4K view of 10M large splats, 337M keys:
// 10.5 against 3.7 ms).  Before the list, the emission expanded each slot's
// candidates, with an atomic per key and a second overlap test for large
// splats: 12.5 ms there, 51 against 18 us on a 1080p view of 1M (1.8M keys),
// 2.3 against 1.35 ms on 64 views of 3M (201M keys).  Counting a batch's
// overlaps per tile in a shared-memory hash table, instead of taking the ranks
// from the frame kernel's atomics, makes that kernel 0.4 ms faster there and
// this one 1.6 ms slower.
constexpr int kEmitUnroll = 4;
constexpr int kEmitBlocksPerSm = 4;
__global__ void __launch_bounds__(kThreads, kEmitBlocksPerSm) emit_bucket_kernel(const __grid_constant__ BucketEmitArgs a)
{
    constexpr int U = kEmitUnroll;
    constexpr int kBatch = kWarps * U;
    __shared__ unsigned long long s_next[2];
    frame_step_begin();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        // straight into host memory: a copy at the frame's end would cost its
        // latency, and nothing after this kernel changes the words
        stamp(a.result, kTimeEmit);
        a.result->total = *a.total;
        a.result->slots = *a.slot_counter;
        a.result->units = *a.unit_count;
        a.result->err = *a.err;
        a.result->overflow = *a.overflow;
    }
    if (*a.overflow || *a.err) {
        // some list was too short, so keys of some tiles were never recorded,
        // or the ranges are meaningless: the host redoes or drops the frame,
        // and until then its tiles are empty
        for (int64_t t = (int64_t)blockIdx.x * kThreads + threadIdx.x; t < 2 * a.tiles; t += (int64_t)gridDim.x * kThreads)
            a.ranges[t] = 0;
        for (int64_t t = (int64_t)blockIdx.x * kThreads + threadIdx.x; a.order && t < a.tiles; t += (int64_t)gridDim.x * kThreads)
            a.order[t] = (int32_t)t;
        if (blockIdx.x == 0 && threadIdx.x == 0) *a.big_count = *a.huge_count = 0u;
        return;
    }
    const int64_t nchunks = (int64_t)(*a.slot_counter >> 32);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (a.order) {
        // tiles before each (group, class)
        static_assert(kOrderClasses == 32, "one class per lane");
        __shared__ int s_before[kMaxRasterGroups * kOrderClasses];
        if (warp == 0) {
            int carry = 0;
            for (int g = 0; g < a.groups; ++g) {
                const int mine = (int)a.class_tiles[g * kOrderClasses + lane];
                int incl = mine;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int t = __shfl_up_sync(kFull, incl, o);
                    if (lane >= o) incl += t;
                }
                s_before[g * kOrderClasses + lane] = carry + incl - mine;
                carry += __shfl_sync(kFull, incl, 31);
            }
        }
        __syncthreads();
        for (int64_t t0 = ((int64_t)blockIdx.x * kWarps + warp) * 32; t0 < a.tiles; t0 += (int64_t)gridDim.x * kThreads) {
            const int64_t t = t0 + lane;
            int cls = -1;
            if (t < a.tiles)
                cls = order_class((uint32_t)(a.ranges[2 * t + 1] - a.ranges[2 * t])) +
                      kOrderClasses * group_of(a.group_tile, a.groups, t);
            const unsigned peers = __match_any_sync(kFull, cls);
            const int leader = __ffs(peers) - 1;
            unsigned head = 0;
            if (cls >= 0 && lane == leader) head = atomicAdd(&a.class_heads[cls], (unsigned)__popc(peers));
            head = __shfl_sync(kFull, head, leader);
            if (cls >= 0) a.order[s_before[cls] + (int)head + __popc(peers & lanemask_lt())] = (int32_t)t;
        }
    }
    if (threadIdx.x == 0) s_next[0] = atomicAdd(a.batch_counter, (unsigned long long)kBatch);
    __syncthreads();
    for (int it = 0;; it ^= 1) {
        const int64_t c0 = (int64_t)s_next[it] + warp * U;
        if ((int64_t)s_next[it] >= nchunks) return;
        // the next batch is on its way while this one is written
        if (threadIdx.x == 0) s_next[it ^ 1] = atomicAdd(a.batch_counter, (unsigned long long)kBatch);
        uint4 h[U];
        uint2 x[U];
        uint32_t slot[U], depth[U];
        int32_t lo[U];
#pragma unroll
        for (int u = 0; u < U; ++u) h[u] = c0 + u < nchunks ? __ldg(&a.chunks[c0 + u]) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if ((h[u].x >> lane) & 1u) x[u] = __ldcs(&a.overlaps[(c0 + u) * 32 + lane]);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if ((h[u].x >> lane) & 1u) {
                const uint32_t owner = x[u].x >> kOverlapTileBits;
                slot[u] = h[u].y + __popc(h[u].z & ((1u << owner) - 1u));
                depth[u] = __ldg(&a.depth[slot[u]]);
                lo[u] = a.ranges[2 * (int64_t)(x[u].x & ((1u << kOverlapTileBits) - 1u))];
            }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if ((h[u].x >> lane) & 1u) {
                a.keys[(int64_t)lo[u] + x[u].y] = ((uint64_t)depth[u] << 32) | slot[u];
            }
        __syncthreads();
    }
}

void launch_emit_bucket(const BucketEmitArgs& a, int num_sms, cudaStream_t st)
{
    const int64_t batch = kWarps * kEmitUnroll;
    const int64_t work = std::max((a.chunk_capacity + batch - 1) / batch, (a.tiles + kThreads - 1) / kThreads);
    const int64_t blocks = std::min<int64_t>(work, (int64_t)num_sms * kEmitBlocksPerSm);
    if (blocks <= 0) return;
    launch_frame_step(emit_bucket_kernel, (unsigned)blocks, kThreads, 0, st, true, a);
}

// ---- 3. sort of the tiles too large for the raster CTAs -------------------------------
//
// Tiles up to the fused capacity are sorted by the raster CTA itself
// (gs_tilesort.cuh).  The larger ones, listed by the tile scan, are sorted
// here beforehand -- up to kTileSortSmemKeys keys by one counting pass in
// shared memory and ranks inside its runs (tilesort::count_sort_tile; the
// radix form of the raster CTA when a run is too long), up to
// kTileSortHugeMax the same in one 1024-thread CTA (above kTileSortHugeKeys in
// parts), else by stable LSD passes through global memory -- and their order is written to `vals` for
// the rasteriser to read.  On the 64-view batch (57k such tiles, 92M keys)
// the counting form takes 1.98 ms against 2.33 ms for the radix form.

namespace {

using tilesort::Smem;

constexpr int kBigThreads = kThreads;

// One stable LSD pass of a tile too large for shared memory, by one CTA:
// digit histogram of the segment, then 4096-key chunks in order, each
// ranked in the block and written at its digits' running starts.
__device__ void global_pass(const uint64_t* in_k, const int32_t* in_v, uint64_t* out_k, int32_t* out_v, const int m,
                            const int shift, const Smem& sm)
{
    constexpr int NT = kBigThreads;
    constexpr int IPT = kTileSortSmemKeys / NT;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool owner = threadIdx.x < 256;
    uint32_t* hist = reinterpret_cast<uint32_t*>(sm.v);  // the value buffer is unused on this path
    if (owner) hist[threadIdx.x] = 0;
    __syncthreads();
    for (int p = threadIdx.x; p < m; p += NT) atomicAdd(&hist[(unsigned)(in_k[p] >> shift) & 0xFFu], 1u);
    __syncthreads();
    const int ex = tilesort::excl_scan<NT>(owner ? (int)hist[threadIdx.x] : 0, sm.scan);
    if (owner) sm.run[threadIdx.x] = ex;
    __syncthreads();
    for (int c0 = 0; c0 < m; c0 += kTileSortSmemKeys) {
        uint64_t k[IPT];
        int32_t v[IPT];
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            const int p = c0 + warp * 32 * IPT + i * 32 + lane;
            if (p < m) {
                k[i] = in_k[p];
                v[i] = in_v ? in_v[p] : (int32_t)(uint32_t)k[i];
            } else {
                k[i] = ~0ull;
                v[i] = 0;
            }
        }
        int pos[IPT];
        tilesort::block_rank<NT, IPT>(k, shift, pos, sm);
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            const int p = c0 + warp * 32 * IPT + i * 32 + lane;
            if (p < m) {
                const unsigned d = (unsigned)(k[i] >> shift) & 0xFFu;
                const int dst = sm.run[d] + (pos[i] - sm.bexcl[d]);
                out_k[dst] = k[i];
                out_v[dst] = v[i];
            }
        }
        __syncthreads();
        if (owner) sm.run[threadIdx.x] += sm.dcount[threadIdx.x];
        __syncthreads();
    }
}

__device__ void sort_tile_global(const TileSortArgs& a, const int64_t start, const int m, const Smem& sm)
{
    constexpr int NT = kBigThreads;
    uint64_t* bk[2] = {a.keys + start, a.keys_alt + start};
    int32_t* bv[2] = {a.vals + start, a.vals_alt + start};
    int cur = 0;
    bool have_v = false;  // values not yet materialised: slot = low key bits

    auto vary_of = [&](const uint64_t hi_mask) {
        uint64_t o = 0, n = ~0ull;
        for (int p = threadIdx.x; p < m; p += NT) {
            const uint64_t x = bk[cur][p];
            o |= x;
            n &= x;
        }
        return tilesort::varying_bits<NT>(o, n, sm.red) & hi_mask;
    };
    auto run_passes = [&](uint64_t mask) {
        while (mask) {
            const int shift = __ffsll((long long)mask) - 1;
            mask &= ~(0xFFull << shift);
            global_pass(bk[cur], have_v ? bv[cur] : nullptr, bk[cur ^ 1], bv[cur ^ 1], m, shift, sm);
            cur ^= 1;
            have_v = true;
        }
    };

    // passes over the top 16 varying depth bits, then the runs of equal
    // prefixes into (depth, index) order (as in the shared-memory sort); the
    // keys keep their slots in the low bits throughout
    int shift;
    run_passes(tilesort::prefix_window(vary_of(0xFFFFFFFF00000000ull), a.prefix_bits, &shift));
    bool too_long = false;
    for (int p = threadIdx.x; p < m; p += NT) too_long |= tilesort::fix_run_at(bk[cur], m, p, shift, a.slot_gi);
    if (!__syncthreads_or(too_long)) {
        // result into a.vals
        for (int p = threadIdx.x; p < m; p += NT) bv[0][p] = (int32_t)(uint32_t)bk[cur][p];
        return;
    }
    // a long run of equal prefixes: sort again on (depth, index), the slots
    // carried as values
    for (int p = threadIdx.x; p < m; p += NT) {
        const uint64_t x = bk[cur][p];
        const int32_t s = (int32_t)(uint32_t)x;
        bv[cur][p] = s;
        bk[cur][p] = (x & 0xFFFFFFFF00000000ull) | (uint32_t)__ldg(&a.slot_gi[s]);
    }
    have_v = true;
    __syncthreads();
    run_passes(vary_of(~0ull));
    if (cur == 1)
        for (int p = threadIdx.x; p < m; p += NT) bv[0][p] = bv[1][p];
}

template <int IPT>
__device__ void sort_big_smem(const TileSortArgs& a, const int64_t start, const int m, const Smem& sm)
{
    tilesort::sort_tile<kBigThreads, IPT>(a.keys + start, m, a.slot_gi, sm, a.prefix_bits);
    for (int p = threadIdx.x; p < m; p += kBigThreads) a.vals[start + p] = (int32_t)(uint32_t)sm.k[p];
}

// The counting form (one placement pass, ranks inside the runs), the
// histogram in the values' part of shared memory; a tile with a long run of
// equal prefixes takes the radix form.
__device__ void sort_big_count(const TileSortArgs& a, const int64_t start, const int m, const Smem& sm)
{
    uint32_t* hist = reinterpret_cast<uint32_t*>(sm.v);
    const bool long_run =
        m <= kBigThreads * 8
            ? tilesort::count_sort_tile<kBigThreads, 8>(a.keys + start, m, a.slot_gi, sm, hist, a.vals + start,
                                                         kTileSortSmemKeys)
            : tilesort::count_sort_tile<kBigThreads, 0>(a.keys + start, m, a.slot_gi, sm, hist, a.vals + start,
                                                         kTileSortSmemKeys);
    if (!long_run) return;
    if (m <= 2048)
        sort_big_smem<8>(a, start, m, sm);
    else
        sort_big_smem<16>(a, start, m, sm);
}

}  // namespace

// Persistent CTAs over the big-tile list.
// 4 blocks per SM (64 registers; the spills are in the radix fallback)
constexpr int kBigBlocksPerSm = 4;
__global__ void __launch_bounds__(kBigThreads, kBigBlocksPerSm) tile_sort_big_kernel(TileSortArgs a)
{
    constexpr int NW = kBigThreads / 32;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int32_t s_bexcl[256];
    __shared__ int32_t s_dcount[256];
    __shared__ int32_t s_run[256];
    __shared__ int32_t s_scan[NW];
    __shared__ uint64_t s_red[2 * NW];
    Smem sm;
    sm.k = reinterpret_cast<uint64_t*>(smem);
    sm.v = reinterpret_cast<int32_t*>(smem + kTileSortSmemKeys * 8);
    sm.whist = reinterpret_cast<uint32_t*>(smem);
    sm.bexcl = s_bexcl;
    sm.dcount = s_dcount;
    sm.scan = s_scan;
    sm.red = s_red;
    sm.run = s_run;
    frame_step_begin();
    const int nbig = (int)*a.big_count;
    for (int j = blockIdx.x; j < nbig; j += gridDim.x) {
        const int64_t t = a.big_list[j];
        const int64_t start = __ldg(&a.ranges[2 * t]);
        const int m = __ldg(&a.ranges[2 * t + 1]) - (int)start;
        if (m <= kTileSortSmemKeys)
            sort_big_count(a, start, m, sm);
        else
            sort_tile_global(a, start, m, sm);
        __syncthreads();  // shared memory is reused by the next tile
    }
}

// The tiles above kTileSortSmemKeys keys, by persistent 1024-thread CTAs
// (one per SM: 128 KB of keys and a 64 KB histogram of 2^15 bins in shared
// memory), in the counting form over 15 depth bits, above kTileSortHugeKeys
// keys in parts.  A tile above kTileSortHugeMax keys, or with a run longer than kMaxRankRun, is handed
// to tile_sort_big_kernel: appended to its list, which that kernel, launched
// after this one on the same stream, reads when it starts.
constexpr int kHugeThreads = 1024;
constexpr int kHugeBits = 15;
__global__ void __launch_bounds__(kHugeThreads, 1) tile_sort_huge_kernel(TileSortArgs a)
{
    constexpr int NW = kHugeThreads / 32;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int32_t s_scan[NW];
    __shared__ uint64_t s_red[2 * NW];
    Smem sm{};
    sm.k = reinterpret_cast<uint64_t*>(smem);
    sm.scan = s_scan;
    sm.red = s_red;
    uint32_t* hist = reinterpret_cast<uint32_t*>(smem + kTileSortHugeKeys * 8);
    frame_step_begin();
    if (blockIdx.x == 0 && threadIdx.x == 0) stamp(a.result, kTimeSort);
    const int nhuge = (int)*a.huge_count;
    for (int j = blockIdx.x; j < nhuge; j += gridDim.x) {
        const int64_t t = a.big_list[a.tiles + j];
        const int64_t start = __ldg(&a.ranges[2 * t]);
        const int m = __ldg(&a.ranges[2 * t + 1]) - (int)start;
        bool handed = m > kTileSortHugeMax;
        if (!handed && m <= kTileSortHugeKeys)
            handed = tilesort::count_sort_tile<kHugeThreads, kTileSortHugeKeys / kHugeThreads, kHugeBits>(
                a.keys + start, m, a.slot_gi, sm, hist, a.vals + start, kTileSortHugeKeys);
        else if (!handed)
            handed = tilesort::count_sort_tile<kHugeThreads, 0, kHugeBits>(a.keys + start, m, a.slot_gi, sm, hist,
                                                                          a.vals + start, kTileSortHugeKeys);
        if (handed && threadIdx.x == 0) a.big_list[atomicAdd(a.big_count, 1u)] = (int32_t)t;
        __syncthreads();  // shared memory is reused by the next tile
    }
}

void launch_tile_sort(const TileSortArgs& a, int num_sms, cudaStream_t st)
{
    constexpr int big_smem = kTileSortSmemKeys * 12;
    constexpr int huge_smem = kTileSortHugeKeys * 12;
    static PerDeviceOnce attr;
    attr.run([] {
        cudaFuncSetAttribute(tile_sort_big_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, big_smem);
        cudaFuncSetAttribute(tile_sort_huge_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, huge_smem);
    });
    if (a.tiles <= 0) return;
    launch_frame_step(tile_sort_huge_kernel, (unsigned)num_sms, kHugeThreads, huge_smem, st, true, a);
    launch_frame_step(tile_sort_big_kernel, (unsigned)(kBigBlocksPerSm * num_sms), kBigThreads, big_smem, st, true, a);
}

}  // namespace gs
