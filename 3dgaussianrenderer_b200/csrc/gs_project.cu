// Per-Gaussian kernels of the gs_b200 pipeline:
//   * stage kernels with the reference's buffer layouts (SH only,
//     projection only), used by the stage API;
//   * the fused frame kernel: SH colour + EWA projection + tile rectangle +
//     exact per-Gaussian overlap count (warp-cooperative) + single-pass
//     decoupled look-back scan of the counts into key offsets, for several
//     views per block so the SH coefficients are read once per group;
//   * the emit kernel that writes (tile|depth, index) keys at those offsets.
#include "gs_kernels.h"

namespace gs {

// ---- stage kernels (reference layouts) -------------------------------------

template <int DEG>
__global__ void __launch_bounds__(256) sh_stage_kernel(int64_t n, const float4* __restrict__ pos,
                                                       const float* __restrict__ sh, int sh_count,
                                                       const ViewParams v, float4* __restrict__ color)
{
    // The grouped SH layout is [group of 256][coefficient][256]; with one
    // Gaussian per thread and 256-thread blocks every coefficient load of a
    // warp is one contiguous 128-byte line (gaussian_render.cu:109-112).
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const float4 p = __ldg(&pos[i]);
    const float3 d = view_dir(v, p);
    const float* base = sh + (int64_t)blockIdx.x * 256 * sh_count + threadIdx.x;
    const float3 c = sh_color<DEG>(d.x, d.y, d.z, base, 256);
    color[i] = make_float4(c.x, c.y, c.z, p.w);
}

__global__ void __launch_bounds__(256) project_stage_kernel(int64_t n, const float4* __restrict__ pos,
                                                            const float4* __restrict__ sr, const ViewParams v,
                                                            float2* __restrict__ xy, float* __restrict__ z,
                                                            float4* __restrict__ ell, float4* __restrict__ conic)
{
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const Splat s = project_gaussian(__ldg(&pos[i]), __ldg(&sr[i]), v);
    xy[i] = make_float2(s.x, s.y);
    z[i] = s.z;
    ell[i] = make_float4(s.cs, s.sn, s.ex, s.ey);
    conic[i] = make_float4(s.ca, s.cb, s.cc, 0.0f);
}

// ---- warp-cooperative overlap counting -------------------------------------
//
// Each lane owns one Gaussian with `cand` candidate tiles.  The warp walks
// the concatenation of its 32 candidate lists 32 candidates at a time, so
// one huge splat does not serialise its lane: lane l tests candidate
// base + l of whichever Gaussian owns it (found by a 5-step search over the
// warp's inclusive scan).

struct WarpCands {
    int incl, excl, total;
};

__device__ __forceinline__ WarpCands warp_scan_cands(const int cand)
{
    const int lane = threadIdx.x & 31;
    int incl = cand;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += t;
    }
    WarpCands w;
    w.incl = incl;
    w.excl = incl - cand;
    w.total = __shfl_sync(kFull, incl, 31);
    return w;
}

__device__ __forceinline__ int owner_of(const int incl, const int c)
{
    int pos = 0;
#pragma unroll
    for (int b = 16; b >= 1; b >>= 1) {
        const int t = __shfl_sync(kFull, incl, pos + b - 1);
        if (t <= c) pos += b;
    }
    return pos;
}

__device__ __forceinline__ unsigned lane_range_mask(const int lo, const int hi)
{
    if (hi <= lo) return 0u;
    const unsigned mhi = hi >= 32 ? kFull : ((1u << hi) - 1u);
    const unsigned mlo = (1u << lo) - 1u;
    return mhi & ~mlo;
}

// Adds a step's ballot to this lane's hits and hit mask.
__device__ __forceinline__ void add_hits(const unsigned bal, const WarpCands& w, const int base, const int cand,
                                         const int c0, int& hits, uint32_t& mask)
{
    const unsigned bits = bal & lane_range_mask(max(w.excl - base, 0), min(w.incl - base, 32));
    if (bits) {
        hits += __popc(bits);
        if (cand <= 32) {
            // lane l of this chunk is walk index base + l - excl of its
            // owner; the walk skips the owner's centre candidate c0
            uint32_t mk = (w.excl >= base) ? (bits >> (w.excl - base)) : (bits << (base - w.excl));
            if (c0 >= 0) {
                const uint32_t low = (1u << c0) - 1u;
                mk = (mk & low) | ((mk & ~low) << 1);
            }
            mask |= mk;
        }
    }
}

// The candidate index in the owner's rectangle of walk index k: the walk
// leaves out the owner's centre candidate oc0 (counted before the walk).
__device__ __forceinline__ int walk_candidate(const int k, const int oc0) { return (oc0 >= 0 && k >= oc0) ? k + 1 : k; }

// The tile holding a splat's centre is a hit (the centre test decides it):
// each lane takes its own before the walk, which then leaves it out -- half
// of the candidates on the benchmark's views.  The tile is found with the tile
// rectangle's own arithmetic and confirmed with the centre test's; a centre on
// a tile border falls through to the walk.  Returns the candidate index, -1
// when there is none; sets the view-local tile.
__device__ __forceinline__ int centre_candidate(const Ell& e, const int4 r, const int cand, const ViewParams& v,
                                                int& tile0)
{
    if (cand <= 0) return -1;
    const int gx = (int)floorf((e.cx + 1.0f) * 0.5f * v.tiles_xf);
    const int gy = (int)floorf((e.cy + 1.0f) * 0.5f * v.tiles_yf);
    const int lx = gx - r.x, ly = gy - r.y;
    if (!(lx >= 0 && lx < r.z && ly >= 0 && ly < r.w && gx >= 0 && gx < v.tiles_x && gy >= 0 && gy < v.tiles_y)) return -1;
    float x0, y0, x1, y1;
    tile_clip_rect(v, gx, gy, x0, y0, x1, y1);
    if (!(e.cx > x0 && e.cx < x1 && e.cy > y0 && e.cy < y1)) return -1;
    tile0 = gy * v.tiles_x + gx;
    return ly * r.z + lx;
}

// The owner's ellipse and rectangle, to the whole warp.
__device__ __forceinline__ void owner_ell(const Ell& e, const int4 r, const int o, Ell& oe, int4& orr)
{
    oe.cx = __shfl_sync(kFull, e.cx, o);
    oe.cy = __shfl_sync(kFull, e.cy, o);
    oe.cs = __shfl_sync(kFull, e.cs, o);
    oe.sn = __shfl_sync(kFull, e.sn, o);
    oe.ex = __shfl_sync(kFull, e.ex, o);
    oe.ey = __shfl_sync(kFull, e.ey, o);
    orr.x = __shfl_sync(kFull, r.x, o);
    orr.y = __shfl_sync(kFull, r.y, o);
    orr.z = __shfl_sync(kFull, r.z, o);
    orr.w = __shfl_sync(kFull, r.w, o);
}

// Returns this lane's number of overlapping tiles; for rectangles of at
// most 32 candidates also the hit mask (bit c = candidate c overlaps).
//
// The overlap test is the reference's, in two phases: the walk decides every
// candidate the cheap evaluation can call, and only if some candidate of the
// warp was too close to call does a second walk settle those in IEEE
// arithmetic, so that the first walk does not hold the IEEE code's registers
// (one walk that calls it 6.81 against 6.25 ms on 64 views of 3M).
__device__ __forceinline__ int warp_count_hits(const Ell& e, const int4 r, const int cand, const ViewParams& v,
                                               uint32_t& mask)
{
    const int lane = threadIdx.x & 31;
    int tile0 = 0;
    const int c0 = centre_candidate(e, r, cand, v, tile0);
    const bool pre = c0 >= 0;
    const WarpCands w = warp_scan_cands(cand - (pre ? 1 : 0));
    int hits = pre ? 1 : 0;
    mask = (pre && cand <= 32) ? (1u << c0) : 0u;
    unsigned undecided = 0;  // this lane's candidates too close to call: bit s of step s, bit 31 of all from 31
    for (int base = 0; base < w.total; base += 32) {
        const int c = base + lane;
        const int o = owner_of(w.incl, c);
        Ell oe;
        int4 orr;
        owner_ell(e, r, o, oe, orr);
        const int oexcl = __shfl_sync(kFull, w.excl, o);
        const int oc0 = __shfl_sync(kFull, c0, o);
        int st = 0;
        int tile = 0;
        if (c < w.total) st = candidate_state(oe, orr, walk_candidate(c - oexcl, oc0), v, tile);
        undecided |= st < 0 ? 1u << min(base >> 5, 31) : 0u;
        add_hits(__ballot_sync(kFull, st > 0), w, base, cand, c0, hits, mask);
    }
    undecided = __reduce_or_sync(kFull, undecided);
    if (undecided) {
        // the steps that hold a candidate too close to call, in IEEE arithmetic
        for (int base = 0; base < w.total; base += 32) {
            if (!((undecided >> min(base >> 5, 31)) & 1u)) continue;
            const int c = base + lane;
            const int o = owner_of(w.incl, c);
            Ell oe;
            int4 orr;
            owner_ell(e, r, o, oe, orr);
            const int oexcl = __shfl_sync(kFull, w.excl, o);
            const int oc0 = __shfl_sync(kFull, c0, o);
            int tile = 0;
            bool hit = false;
            const int oc = walk_candidate(c - oexcl, oc0);
            if (c < w.total && candidate_state(oe, orr, oc, v, tile) < 0) hit = candidate_hit_ieee(oe, tile, v);
            const unsigned bal = __ballot_sync(kFull, hit);
            if (bal) add_hits(bal, w, base, cand, c0, hits, mask);
        }
    }
    return hits;
}

// ---- overlaps of a warp's Gaussians, for the tile buckets -------------------------
//
// The same walk, but every overlap is recorded once and for all: one atomic on
// its tile's key count returns its rank in the tile, and (tile, owner lane,
// rank) goes to the overlap list in chunks of 32 (BucketEmitArgs).  The bucket
// emission then needs neither another overlap test nor atomics.  An atomic's
// result is used one step of the walk later, so its latency overlaps the next
// step's tests.
//
// Every lane with candidates takes a slot; slots and chunks come from one
// 64-bit atomic per warp (slots in the low half): a chunk for the centre tiles
// and one per step of the walk, the step's ballot being its mask.  Splats of
// more than kLargeCandidates candidates are left to large_overlap_kernel, so a
// walk has at most 32 steps and lane s keeps step s's ballot until the chunks
// are written.  The walk's registers bound the frame kernel (64 per thread):
// what the lanes exchange is packed.

// A warp's walk before its first step; the slots and chunks and the centre
// tiles' ranks are on their way.
struct BucketWalk {
    int incl;                // inclusive scan of the lanes' candidates but the centre
    int total;
    int own;                 // (exclusive scan << 8 | centre candidate + 1) of this lane
    unsigned preb;           // lanes with a centre tile
    unsigned long long got;  // lane 0: (first chunk << 32 | first slot)
};

// Overlaps recorded but not yet written, because their ranks (and for the
// first ones their chunk) are on their way: lanes with `has` write (where, rank
// of lane `from` + more).
struct OverlapPending {
    uint32_t where;  // tile | owner << kOverlapTileBits
    uint32_t rank;
    int from, more;
    bool has;
};

__device__ __forceinline__ void write_pending(const FrameArgs& a, const OverlapPending& x, const uint32_t chunk)
{
    const uint32_t rank = __shfl_sync(kFull, x.rank, x.from) + (uint32_t)x.more;
    // chunks past the list's end are dropped: the frame is redone with a longer one
    if (x.has && chunk < a.chunk_capacity)
        a.overlaps[(int64_t)chunk * 32 + (threadIdx.x & 31)] = make_uint2(x.where, rank);
}

// The candidate of this lane in step `s` of the walk: 1 hit, 0 miss, -1 too
// close to call; sets its owner, the owner's ellipse and the view-local tile.
__device__ __forceinline__ int walk_step(const Ell& e, const int2 pr, const BucketWalk& k, const int s, const ViewParams& v,
                                         Ell& oe, int& o, int& tile)
{
    const int c = 32 * s + (int)(threadIdx.x & 31);
    o = owner_of(k.incl, c);
    oe.cx = __shfl_sync(kFull, e.cx, o);
    oe.cy = __shfl_sync(kFull, e.cy, o);
    oe.cs = __shfl_sync(kFull, e.cs, o);
    oe.sn = __shfl_sync(kFull, e.sn, o);
    oe.ex = __shfl_sync(kFull, e.ex, o);
    oe.ey = __shfl_sync(kFull, e.ey, o);
    int2 opr;
    opr.x = __shfl_sync(kFull, pr.x, o);
    opr.y = __shfl_sync(kFull, pr.y, o);
    const int own = __shfl_sync(kFull, k.own, o);
    tile = 0;
    if (c >= k.total) return 0;
    return candidate_state(oe, unpack_rect(opr), walk_candidate(c - (own >> 8), (own & 0xFF) - 1), v, tile);
}

// Sets up the walk over the candidates (cand, 0 for lanes that take no part)
// of a warp whose lanes in `owners` take slots, and counts the centre tiles.
__device__ __forceinline__ BucketWalk start_walk(const Ell& e, const int4 r, const int cand, const ViewParams& v,
                                                 const FrameArgs& a, const unsigned owners, OverlapPending& x)
{
    const int lane = threadIdx.x & 31;
    BucketWalk k;
    int tile0 = 0;
    const int c0 = centre_candidate(e, r, cand, v, tile0);
    x.has = c0 >= 0;
    k.preb = __ballot_sync(kFull, x.has);
    const WarpCands w = warp_scan_cands(cand - (x.has ? 1 : 0));
    k.incl = w.incl;
    k.total = w.total;
    k.own = (w.excl << 8) | (c0 + 1);
    k.got = 0;
    if (lane == 0)
        k.got = atomicAdd(a.slot_counter, ((unsigned long long)((k.preb ? 1 : 0) + ((w.total + 31) >> 5)) << 32) |
                                              (unsigned long long)__popc(owners));
    // neighbours in the scene's order mostly share their centre tile: one
    // atomic per tile and warp (1024x1024 view of 3M: frame kernel -14 %)
    x.where = ((uint32_t)v.tile_offset + (uint32_t)tile0) | ((uint32_t)lane << kOverlapTileBits);
    x.rank = 0;
    x.from = lane;
    x.more = 0;
    if (x.has) {
        const unsigned grp = __match_any_sync(k.preb, tile0);
        x.from = __ffs(grp) - 1;
        x.more = __popc(grp & lanemask_lt());
        if (lane == x.from) x.rank = atomicAdd(&a.tile_count[v.tile_offset + tile0], (unsigned)__popc(grp));
    }
    return k;
}

// The walk.  Leaves the overlaps of its last step (or of the centre tiles) in
// `x`, to be written to chunk `last`.  With `track`, returns the lanes that own
// an overlap.
__device__ __forceinline__ unsigned run_walk(const Ell& e, const int2 pr, const ViewParams& v, const FrameArgs& a,
                                             const BucketWalk& k, const bool track, OverlapPending& x, unsigned& mine)
{
    const int lane = threadIdx.x & 31;
    const uint32_t toff = (uint32_t)v.tile_offset;
    const int steps = (k.total + 31) >> 5;
    unsigned reached = k.preb;
    uint32_t chunk = 0;  // of the pending overlaps
    unsigned undecided = 0;  // this lane's candidates too close to call: bit s of step s
    mine = 0;
    for (int s = 0; s < steps; ++s) {
        int o, tile;
        Ell oe;
        const int st = walk_step(e, pr, k, s, v, oe, o, tile);
        undecided |= st < 0 ? 1u << s : 0u;
        const bool hit = st > 0;
        const unsigned bal = __ballot_sync(kFull, hit);
        if (lane == s) mine = bal;
        if (track) reached |= __reduce_or_sync(kFull, hit ? 1u << o : 0u);
        uint32_t rank = 0;
        if (hit) rank = atomicAdd(&a.tile_count[toff + (uint32_t)tile], 1u);
        if (s == 0) chunk = (uint32_t)(__shfl_sync(kFull, k.got, 0) >> 32);
        if (s > 0 || k.preb) write_pending(a, x, chunk++);
        x = {(toff + (uint32_t)tile) | ((uint32_t)o << kOverlapTileBits), rank, lane, 0, hit};
    }
    undecided = __reduce_or_sync(kFull, undecided);
    if (undecided) {
        // the steps that hold a candidate too close to call, in IEEE arithmetic.
        // Walking all steps again doubled the time of such a warp, and a frame
        // of one wave waits for its longest (to the emission, 100k Gaussians 56
        // -> 47 us; 64 views of 3M 6.28 -> 5.89 ms).
        write_pending(a, x, chunk);
        x.has = false;
        const uint32_t chunk0 = chunk - (uint32_t)(steps - 1);
        for (; undecided; undecided &= undecided - 1) {
            const int s = __ffs(undecided) - 1;
            int o, tile;
            Ell oe;
            bool hit = walk_step(e, pr, k, s, v, oe, o, tile) < 0;
            if (hit) hit = candidate_hit_ieee(oe, tile, v);
            const unsigned bal = __ballot_sync(kFull, hit);
            if (lane == s) mine |= bal;
            if (track) reached |= __reduce_or_sync(kFull, hit ? 1u << o : 0u);
            OverlapPending y = {(toff + (uint32_t)tile) | ((uint32_t)o << kOverlapTileBits), 0u, lane, 0, hit};
            if (hit) y.rank = atomicAdd(&a.tile_count[toff + (uint32_t)tile], 1u);
            write_pending(a, y, chunk0 + (uint32_t)s);
        }
    }
    return reached;
}

// ---- large splats -----------------------------------------------------------------
//
// A splat that covers hundreds of tiles would hold its warp, and its block,
// while the rest of the frame is long done: on a 4K view of 10M large splats the
// frame kernel spent 60 % of its time in the few blocks next to the camera.
// Splats of more than kLargeCandidates candidates keep their ellipse and
// rectangle at their slot and are listed, their candidates cut into units of
// kUnitCandidates; large_overlap_kernel takes one unit per warp, from a
// counter.  The threshold is about where a splat fills whole steps of a warp
// of its own.

// Lists the units of this warp's large splats.
__device__ __forceinline__ void list_large(const int cand, const bool large, const uint32_t slot, const FrameArgs& a)
{
    const int units = large ? (cand + kUnitCandidates - 1) / kUnitCandidates : 0;
    const WarpCands w = warp_scan_cands(units);
    unsigned long long got = 0;
    if ((threadIdx.x & 31) == 0) got = atomicAdd(a.unit_count, (unsigned long long)w.total);
    const int64_t u0 = (int64_t)__shfl_sync(kFull, got, 0) + w.excl;
    for (int u = 0; u < units; ++u)
        if (u0 + u < a.unit_capacity) a.units[u0 + u] = make_uint2(slot, (uint32_t)u);
}

// One unit per warp: its overlaps' ballots first (step s's in lane s), then
// exactly as many chunks as they fill, then the ranks and the list entries.
__global__ void __launch_bounds__(256) large_overlap_kernel(const __grid_constant__ FrameArgs a)
{
    static_assert(kUnitCandidates == 1024, "one step of a unit per lane");
    const int lane = threadIdx.x & 31;
    frame_step_begin();
    int64_t units = (int64_t)*a.unit_count;
    if (units > a.unit_capacity) units = a.unit_capacity;
    if (units == 0) return;
    // a warp's first unit is its own number, the next ones come from the counter
    const int64_t warps = (int64_t)gridDim.x * 8;
    int64_t k = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    for (unsigned long long next = 0; k < units; k = warps + (int64_t)__shfl_sync(kFull, next, 0)) {
        if (lane == 0) next = atomicAdd(a.unit_counter, 1ull);  // on its way while this unit is walked
        const uint2 unit = a.units[k];
        const uint32_t slot = unit.x;
        const float2 centre = __ldg(&a.xy[slot]);
        const float4 el = __ldg(&a.ell[slot]);
        const Ell e = {centre.x, centre.y, el.x, el.y, el.z, el.w};
        const int4 r = unpack_rect(__ldg(&a.rect[slot]));
        const ViewParams& v = a.views[(uint32_t)__ldg(&a.offsets[slot]) / (uint32_t)a.n];
        const int c0 = (int)unit.y * kUnitCandidates;
        const int total = min(rect_candidates(r) - c0, kUnitCandidates);
        const int steps = (total + 31) >> 5;
        unsigned mine = 0;
        for (int s = 0; s < steps; ++s) {
            const int c = 32 * s + lane;
            int tile;
            const bool hit = c < total && candidate_hit(e, r, c0 + c, v, tile);
            const unsigned bal = __ballot_sync(kFull, hit);
            if (lane == s) mine = bal;
        }
        const WarpCands w = warp_scan_cands(__popc(mine));
        if (w.total == 0) continue;
        const int chunks = (w.total + 31) >> 5;
        unsigned long long got = 0;
        if (lane == 0) got = atomicAdd(a.slot_counter, (unsigned long long)chunks << 32);
        const int64_t first = (int64_t)(__shfl_sync(kFull, got, 0) >> 32);
        const bool room = first + chunks <= a.chunk_capacity;
        if (room && lane < chunks) {
            const int left = w.total - 32 * lane;
            a.chunks[first + lane] = make_uint4(left >= 32 ? kFull : (1u << left) - 1u, slot, 0u, 0u);
        }
        for (int s0 = 0; s0 < steps; s0 += 4) {
            uint2 x[4];
            int at[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int s = s0 + u;
                const unsigned bal = s < steps ? __shfl_sync(kFull, mine, s & 31) : 0u;
                at[u] = __shfl_sync(kFull, w.excl, s & 31) + __popc(bal & lanemask_lt());
                if (!((bal >> lane) & 1u)) {
                    at[u] = -1;
                    continue;
                }
                int lx, ly;
                divmod_small(c0 + 32 * s + lane, r.z, ly, lx);
                x[u].x = (uint32_t)v.tile_offset + (uint32_t)((r.y + ly) * v.tiles_x + r.x + lx);
                x[u].y = atomicAdd(&a.tile_count[x[u].x], 1u);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (room && at[u] >= 0) a.overlaps[first * 32 + at[u]] = x[u];
        }
    }
}

// ---- block scan + decoupled look-back along one chain ---------------------------

// This thread's exclusive offset within a chain of blocks (`status[0..len)`,
// block `link` of it); the last block of the chain writes the chain total.
__device__ __forceinline__ int64_t chain_offsets(const int hits, uint64_t* status, const int64_t link,
                                                 const int64_t len, const uint32_t epoch, int64_t* chain_total,
                                                 int* err)
{
    __shared__ int s_warp[8];
    __shared__ int64_t s_base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = hits;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int k = 0; k < 8; ++k) {
            const int t = s_warp[k];
            s_warp[k] = run;
            run += t;
        }
        const uint64_t agg = (uint64_t)run;
        uint64_t excl = 0;
        if (link == 0) {
            store_status(status, status_word(kFlagP, epoch, agg));
        } else {
            store_status(status + link, status_word(kFlagA, epoch, agg));
            excl = look_back(status, link, 1, epoch, err, kErrTimeout);
            store_status(status + link, status_word(kFlagP, epoch, excl + agg));
        }
        s_base = (int64_t)excl;
        if (link == len - 1) *chain_total = (int64_t)(excl + agg);
    }
    __syncthreads();
    const int64_t r = s_base + s_warp[warp] + (incl - hits);
    __syncthreads();  // s_warp / s_base are reused by the next call
    return r;
}

__device__ __forceinline__ int64_t acquire_tile(unsigned long long* counter)
{
    __shared__ int64_t s_tile;
    if (threadIdx.x == 0) s_tile = (int64_t)atomicAdd(counter, 1ull);
    __syncthreads();
    const int64_t t = s_tile;
    return t;
}

// ---- fused frame kernel ------------------------------------------------------

//
// Block `tile` (taken in dynamic order, so a look-back only ever waits on a
// block that is already running) owns group g = tile % groups for views
// [c*vpb, (c+1)*vpb), c = tile / groups.  It reads position and
// scale/rotation of its 256 Gaussians once and, for SH scenes, brings the
// group's coefficients (the first 3*(DEG+1)^2 rows of the grouped layout,
// contiguous) into shared memory with one TMA bulk copy, once a view shows one
// of them.  Then per view:
// SH colour, projection, tile rectangle, exact overlap count, and the
// within-view key offset from that view's look-back chain.  Gaussians that
// overlap no tile write only their offset.
//
// BUCKET: no scan at all -- each (view, Gaussian) with candidate tiles takes a
// slot and its overlaps go to the overlap list with their ranks in their
// tiles (start_walk, run_walk); the blocks are independent and run in launch order.
__device__ __forceinline__ void sh_wait(uint64_t* bar, int* err)
{
    int spins = 0;
    while (!mbar_try_wait(bar, 0)) {
        if (++spins > kSpinLimit) {
            // a bulk copy from valid device memory always lands; report and
            // carry on (the frame is discarded by the host)
            atomicCAS(err, 0, kErrTimeout);
            return;
        }
    }
}

// A load the compiler may not keep in registers across the views.
__device__ __forceinline__ float4 reload(const float4* p)
{
    float4 x;
    asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w)
                 : "l"(p));
    return x;
}

// The T_min raster record of a splat: centre from e, conic in (g.x, g.y, g.z).
__device__ __forceinline__ void write_record(float4* rec, const Ell& e, const float4 g, const float4 col)
{
    float ex, ey, A = -0.72134752f * g.x, B = -1.44269504f * g.y, C = -0.72134752f * g.z;
    float L = lg2_approx(col.w);
    const float det = g.x * g.z - g.y * g.y;
    if (!(det > 0.0f) || !(g.x > 0.0f) || !(g.z > 0.0f) || !(col.w > kCullAlpha)) {
        // contributes nothing anywhere: alpha below the cutoff, or a conic
        // that is not positive definite
        ex = ey = -1e30f;
        A = B = C = 0.0f;
        L = -1e30f;
    } else {
        // qc = 2 ln(opacity / cutoff) = 2 ln 2 (L + 18); 1.0001 covers the
        // approximations
        const float qc = 1.38643f * (L + 18.0f);
        const float rdet = rcp_approx(det);
        ex = sqrt_approx(qc * g.z * rdet);
        ey = sqrt_approx(qc * g.x * rdet);
    }
    rec[0] = make_float4(e.cx, e.cy, ex, ey);
    rec[1] = make_float4(A, B, C, L);
    rec[2] = make_float4(col.x, col.y, col.z, 0.0f);
}

// MANY: a block draws several views.  It then keeps its Gaussians' attributes
// in registers and waits for their coefficients once, before the first view;
// with one view the attributes are read again after the walk, which needs the
// registers, and the copy is asked for only where a Gaussian is in view and
// overlaps the walk (1080p view of 1M: 104 against 112 us; 64 views of 3M: 6.3
// against 6.6 ms).
// Blocks per SM: 4 (64 registers, at which the SH bucket forms spill 56 to 64
// bytes a thread); the exact projection at SH degree 3 keeps 80 registers
// (3 blocks)
template <int DEG, bool BUCKET, bool FAST, bool MANY>
__global__ void __launch_bounds__(256, (DEG >= 3 && !FAST) ? 3 : 4) frame_project_kernel(const __grid_constant__ FrameArgs a)
{
    extern __shared__ __align__(128) float s_sh[];  // [3*(DEG+1)^2][256]
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ float4 s_geom[BUCKET ? 256 : 1];  // conic and depth across the walk
    const int64_t tile = BUCKET ? (int64_t)blockIdx.x : acquire_tile(a.tile_counter);
    const int64_t chunk = tile / a.groups;
    const int64_t group = tile - chunk * a.groups;
    const int i = (int)group * 256 + (int)threadIdx.x;  // n < 2^31
    const bool valid = i < a.n;
    const int v0 = (int)chunk * a.views_per_block;
    const int v1 = min(a.num_views, v0 + a.views_per_block);
    const uint32_t epoch = a.epoch_dev ? *a.epoch_dev : a.epoch;
    constexpr int NCOEF = DEG >= 0 ? 3 * (DEG + 1) * (DEG + 1) : 0;
    const int at = valid ? i : 0;  // where this thread's loads go
    int gid = i;  // the Gaussian's caller index: equal depths are ordered by it
    if (BUCKET && a.orig) gid = __ldg(&a.orig[at]);

    if (BUCKET) frame_step_begin();
    if (BUCKET && blockIdx.x == 0 && threadIdx.x == 0) stamp(a.result, kTimeStart);
    if (BUCKET && blockIdx.x == 0)
        for (int k = threadIdx.x; k < a.zero_count; k += 256) a.zero_words[k] = 0u;
    if (DEG >= 0 && threadIdx.x == 0) mbar_init(&s_bar, 1);
    bool sh_asked = DEG < 0 || MANY;  // the coefficients' copy has started (block-uniform) ...
    bool sh_here = sh_asked;          // ... and, as this thread knows, landed
    auto ask_sh = [&] {
        bulk_load(s_sh, a.sh + group * 256 * (int64_t)a.sh_count, NCOEF * 256 * sizeof(float), &s_bar);
    };
    float4 kept_p = make_float4(0.f, 0.f, 0.f, 0.f), kept_sr = kept_p;
    if (MANY) {
        if (DEG >= 0 && threadIdx.x == 0) ask_sh();
        kept_p = __ldg(&a.pos[at]);
        kept_sr = __ldg(&a.sr[at]);
        if (DEG >= 0) {
            __syncthreads();  // barrier initialised before anyone polls it
            sh_wait(&s_bar, a.err);
        }
    }

    // the colour towards view v: of the model, or from the coefficients
    auto colour = [&](const ViewParams& v) {
        if (DEG < 0) return reload(&a.color_in[at]);
        if (!sh_here) sh_wait(&s_bar, a.err);
        sh_here = true;
        const float4 p = MANY ? kept_p : reload(&a.pos[at]);
        const float3 d = view_dir(v, p);
        const float3 c = sh_color<(DEG < 0 ? 0 : DEG), false>(d.x, d.y, d.z, s_sh + threadIdx.x, 256);
        return make_float4(c.x, c.y, c.z, p.w);
    };

    for (int view = v0; view < v1; ++view) {
        const ViewParams& v = a.views[view];
        Ell e = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        int4 r = make_int4(0, 0, 0, 0);
        int cand = 0;
        Splat s;
        bool projected = false;
        if (valid) {
            // outside the frustum: culled, no tile (whole warps of a
            // spatially ordered scene skip the projection together)
            const float4 p = MANY ? kept_p : reload(&a.pos[at]), sr = MANY ? kept_sr : reload(&a.sr[at]);
            const ViewPos w = view_position<FAST>(p, v);
            if (in_frustum(w)) {
                projected = true;
                s = project_gaussian<FAST>(w, sr, v);
                e = {s.x, s.y, s.cs, s.sn, s.ex, s.ey};
                r = tile_rect(e, v);
                cand = rect_candidates(r);
            }
        }
        if (!sh_asked) {
            // the barrier also publishes s_bar
            sh_asked = __syncthreads_or(cand > 0) != 0;
            if (sh_asked && threadIdx.x == 0) ask_sh();
        }
        if (a.probe_xy && valid) {
            const int64_t q = (int64_t)view * a.n + gid;
            a.probe_xy[q] = projected ? make_float2(s.x, s.y) : make_float2(-128.0f, -128.0f);
            a.probe_z[q] = projected ? s.z : -128.0f;
            a.probe_ell[q] = projected ? make_float4(s.cs, s.sn, s.ex, s.ey) : make_float4(0.f, 0.f, 0.f, 0.f);
            a.probe_conic[q] = projected ? make_float4(s.ca, s.cb, s.cc, 0.0f) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        // the overlap test is the reference's in every mode: the tile lists
        // of the projected floats are exactly those of the reference's build
        if constexpr (BUCKET) {
            const unsigned owners = __ballot_sync(kFull, cand > 0);
            if (owners == 0) continue;  // warp-uniform
            const bool large = cand > kLargeCandidates;
            OverlapPending x;
            const BucketWalk k = start_walk(e, r, large ? 0 : cand, v, a, owners, x);
            const int2 pr = pack_rect(r);
            // what the walk has no registers for
            if (cand > 0) s_geom[threadIdx.x] = make_float4(s.ca, s.cb, s.cc, s.z);
            unsigned mine;
            const unsigned reached = run_walk(e, pr, v, a, k, a.probe_color != nullptr, x, mine);
            const unsigned long long got = __shfl_sync(kFull, k.got, 0);
            const uint32_t o = (uint32_t)got + (uint32_t)__popc(owners & lanemask_lt());
            if (cand > 0) {
                const float4 g = s_geom[threadIdx.x];
                a.offsets[o] = view * (int32_t)a.n + gid;
                a.depth[o] = depth_bits(g.w);
                if (large) {
                    a.rect[o] = pr;
                    a.ell[o] = make_float4(e.cs, e.sn, e.ex, e.ey);
                }
                if (a.raster_mode == 0 || large) a.xy[o] = make_float2(e.cx, e.cy);
                // the colour only matters for items that can reach a tile
                const float4 col = colour(v);
                if (a.raster_mode == 0) {
                    a.conic[o] = make_float4(g.x, g.y, g.z, 0.0f);
                    a.color[o] = col;
                } else {
                    write_record(a.rec + 3 * (int64_t)o, e, g, col);
                }
                if (a.probe_color) {
                    // a large splat reaches a tile unless an extent is zero
                    // (ellipse_rect_overlap_clear) and its centre is on a border
                    int t0;
                    const bool hit = large ? (e.ex != 0.0f && e.ey != 0.0f) ||
                                                 centre_candidate(e, unpack_rect(pr), cand, v, t0) >= 0
                                           : ((reached >> (threadIdx.x & 31)) & 1u) != 0;
                    if (hit) a.probe_color[(int64_t)view * a.n + gid] = col;
                }
            }
            const int lane = threadIdx.x & 31, steps = (k.total + 31) >> 5;
            const uint32_t chunk = (uint32_t)(got >> 32) + (k.preb ? 1u : 0u);  // of step 0
            write_pending(a, x, chunk + (uint32_t)steps - 1u);
            if (lane < steps && chunk + (uint32_t)lane < a.chunk_capacity)
                a.chunks[chunk + (uint32_t)lane] = make_uint4(mine, (uint32_t)got, owners, 0u);
            if (lane == 0 && k.preb && chunk - 1u < a.chunk_capacity)
                a.chunks[chunk - 1u] = make_uint4(k.preb, (uint32_t)got, owners, 0u);
            if (__any_sync(kFull, large)) list_large(cand, large, o, a);
        } else {
            uint32_t mask;
            const int hits = warp_count_hits(e, r, cand, v, mask);
            const int64_t off = chain_offsets(hits, a.status + (int64_t)view * a.groups, group, a.groups, epoch,
                                              a.view_total + view, a.err);
            const int64_t o = (int64_t)view * a.n + i;
            if (valid) a.offsets[o] = (int32_t)off;
            if (hits > 0) {
                const float4 col = colour(v);
                a.z[o] = s.z;
                a.rect[o] = pack_rect(r);
                a.hitmask[o] = mask;
                if (cand > 32) a.ell[o] = make_float4(s.cs, s.sn, s.ex, s.ey);
                if (a.raster_mode == 0 || cand > 32) a.xy[o] = make_float2(s.x, s.y);
                if (a.raster_mode == 0) {
                    a.color[o] = col;
                    a.conic[o] = make_float4(s.ca, s.cb, s.cc, 0.0f);
                } else {
                    write_record(a.rec + 3 * o, e, make_float4(s.ca, s.cb, s.cc, s.z), col);
                }
            }
        }
    }
    // the copy lands before the block's shared memory goes to another one
    if (DEG >= 0 && threadIdx.x == 0 && sh_asked && !sh_here) sh_wait(&s_bar, a.err);
}

// Count-only variant for the stage API: rectangle + exact count + scan from
// already projected (xy, ellipse) in the reference layouts (one view).
__global__ void __launch_bounds__(256) count_stage_kernel(FrameArgs a)
{
    const int64_t tile = acquire_tile(a.tile_counter);
    const int64_t i = tile * 256 + threadIdx.x;
    const bool valid = i < a.n;
    const ViewParams& v = a.views[0];
    Ell e = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    int4 r = make_int4(0, 0, 0, 0);
    int cand = 0;
    if (valid) {
        const float2 c = __ldg(&a.xy[i]);
        const float4 el = __ldg(&a.ell[i]);
        e = {c.x, c.y, el.x, el.y, el.z, el.w};
        r = tile_rect(e, v);
        cand = rect_candidates(r);
        a.rect[i] = pack_rect(r);
    }
    uint32_t mask;
    const int hits = warp_count_hits(e, r, cand, v, mask);
    const int64_t off = chain_offsets(hits, a.status, tile, a.groups, a.epoch, a.view_total, a.err);
    if (valid) {
        a.offsets[i] = (int32_t)off;
        a.hitmask[i] = mask;
    }
}

__global__ void view_base_kernel(const int64_t* view_total, int num_views, int64_t* view_base, int64_t* total)
{
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        int64_t run = 0;
        for (int v = 0; v < num_views; ++v) {
            view_base[v] = run;
            run += view_total[v];
        }
        *total = run;
    }
}

// ---- emit -------------------------------------------------------------------
//
// Rewalks each warp's candidates and writes every hit at
// view_base + offsets[g] + (number of earlier hits of g), so keys leave in
// (view, Gaussian) order with tiles ascending inside a Gaussian; a stable
// sort then breaks equal keys by index.  The key holds the global tile id
// (view tile offset + tile), the value the view-flattened Gaussian index.
__global__ void __launch_bounds__(256) emit_kernel(EmitArgs a)
{
    const int64_t gi = (int64_t)blockIdx.x * 256 + threadIdx.x;  // over views * n
    const int64_t total_items = (int64_t)a.num_views * a.n;
    const bool valid = gi < total_items;
    // a warp may straddle two views; every owner's view travels with it
    const int view = valid ? (int)(gi / a.n) : 0;
    const int lane = threadIdx.x & 31;

    int cand = 0, hits = 0;
    int4 r = make_int4(0, 0, 0, 0);
    Ell e = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    float depth = 0.f;
    int64_t off = 0;
    if (valid) {
        const int64_t i = gi - (int64_t)view * a.n;
        const int64_t own = a.offsets[gi];
        const int64_t next = (i + 1 < a.n) ? (int64_t)a.offsets[gi + 1] : a.view_total[view];
        hits = (int)(next - own);
        off = a.view_base[view] + own;
        if (hits > 0) {
            r = unpack_rect(a.rect[gi]);
            cand = rect_candidates(r);
            depth = a.z[gi];
            if (cand <= 32 && a.hitmask) {
                // the counting pass recorded which candidates overlap: expand
                // the mask in candidate order, no overlap test needed
                const ViewParams& v = a.views[view];
                uint32_t m = a.hitmask[gi];
                int64_t dst = off;
                while (m) {
                    const int c = __ffs(m) - 1;
                    m &= m - 1;
                    int ly, lx;
                    divmod_small(c, r.z, ly, lx);
                    const int gx = r.x + lx, gy = r.y + ly;
                    if (dst < a.capacity) {
                        a.keys[dst] = make_key((uint64_t)(v.tile_offset + gy * v.tiles_x + gx), depth);
                        a.values[dst] = (int32_t)gi;
                    }
                    ++dst;
                }
                cand = 0;  // done: stays out of the cooperative walk
            } else {
                const float2 c = a.xy[gi];
                const float4 el = a.ell[gi];
                e = {c.x, c.y, el.x, el.y, el.z, el.w};
            }
        }
    }
    // rectangles with more than 32 candidates: the warp walks them together
    if (__ballot_sync(kFull, cand > 0) == 0) return;
    const WarpCands w = warp_scan_cands(cand);
    int running = 0;
    for (int base = 0; base < w.total; base += 32) {
        const int c = base + lane;
        const int o = owner_of(w.incl, c);
        Ell oe;
        oe.cx = __shfl_sync(kFull, e.cx, o);
        oe.cy = __shfl_sync(kFull, e.cy, o);
        oe.cs = __shfl_sync(kFull, e.cs, o);
        oe.sn = __shfl_sync(kFull, e.sn, o);
        oe.ex = __shfl_sync(kFull, e.ex, o);
        oe.ey = __shfl_sync(kFull, e.ey, o);
        int4 orr;
        orr.x = __shfl_sync(kFull, r.x, o);
        orr.y = __shfl_sync(kFull, r.y, o);
        orr.z = __shfl_sync(kFull, r.z, o);
        orr.w = __shfl_sync(kFull, r.w, o);
        const int oexcl = __shfl_sync(kFull, w.excl, o);
        const int oincl = __shfl_sync(kFull, w.incl, o);
        const int orun = __shfl_sync(kFull, running, o);
        const float oz = __shfl_sync(kFull, depth, o);
        const long long ooff = __shfl_sync(kFull, (long long)off, o);
        const int oview = __shfl_sync(kFull, view, o);
        bool hit = false;
        int tile = 0;
        if (c < w.total)
            hit = candidate_hit(oe, orr, c - oexcl, a.views[oview], tile);
        const unsigned bal = __ballot_sync(kFull, hit);
        if (hit) {
            const unsigned omask = lane_range_mask(max(oexcl - base, 0), min(oincl - base, 32));
            const int rank = __popc(bal & omask & lanemask_lt());
            const int64_t dst = ooff + orun + rank;
            if (dst < a.capacity) {
                const int64_t gtile = a.views[oview].tile_offset + tile;
                a.keys[dst] = make_key((uint64_t)gtile, oz);
                a.values[dst] = (int32_t)((int64_t)blockIdx.x * 256 + (threadIdx.x & ~31) + o);
            }
        }
        running += __popc(bal & lane_range_mask(max(w.excl - base, 0), min(w.incl - base, 32)));
    }
}

// ---- launchers ----------------------------------------------------------------

void launch_sh_stage(int64_t n, const float4* pos, const float* sh, int sh_count, int deg, const ViewParams& v,
                     float4* color, cudaStream_t st)
{
    const unsigned grid = (unsigned)((n + 255) / 256);
    if (grid == 0) return;
    switch (deg) {
        case 0: sh_stage_kernel<0><<<grid, 256, 0, st>>>(n, pos, sh, sh_count, v, color); break;
        case 1: sh_stage_kernel<1><<<grid, 256, 0, st>>>(n, pos, sh, sh_count, v, color); break;
        case 2: sh_stage_kernel<2><<<grid, 256, 0, st>>>(n, pos, sh, sh_count, v, color); break;
        default: sh_stage_kernel<3><<<grid, 256, 0, st>>>(n, pos, sh, sh_count, v, color); break;
    }
}

void launch_project_stage(int64_t n, const float4* pos, const float4* sr, const ViewParams& v, float2* xy,
                          float* z, float4* ell, float4* conic, cudaStream_t st)
{
    const unsigned grid = (unsigned)((n + 255) / 256);
    if (grid == 0) return;
    project_stage_kernel<<<grid, 256, 0, st>>>(n, pos, sr, v, xy, z, ell, conic);
}

template <int DEG, bool BUCKET, bool FAST, bool MANY>
static void launch_frame_views(const FrameArgs& a, cudaStream_t st)
{
    constexpr int NCOEF = DEG >= 0 ? 3 * (DEG + 1) * (DEG + 1) : 0;
    constexpr int smem = NCOEF * 256 * (int)sizeof(float);
    static PerDeviceOnce attr;
    attr.run([] {
        cudaFuncSetAttribute(frame_project_kernel<DEG, BUCKET, FAST, MANY>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    });
    frame_project_kernel<DEG, BUCKET, FAST, MANY><<<(unsigned)a.num_tiles, 256, smem, st>>>(a);
}

template <int DEG, bool BUCKET, bool FAST>
static void launch_frame_deg(const FrameArgs& a, cudaStream_t st)
{
    if (a.views_per_block > 1)
        launch_frame_views<DEG, BUCKET, FAST, true>(a, st);
    else
        launch_frame_views<DEG, BUCKET, FAST, false>(a, st);
}

template <bool BUCKET, bool FAST>
static void launch_frame_mode(const FrameArgs& a, int deg, cudaStream_t st)
{
    switch (deg) {
        case -1: launch_frame_deg<-1, BUCKET, FAST>(a, st); break;
        case 0: launch_frame_deg<0, BUCKET, FAST>(a, st); break;
        case 1: launch_frame_deg<1, BUCKET, FAST>(a, st); break;
        case 2: launch_frame_deg<2, BUCKET, FAST>(a, st); break;
        default: launch_frame_deg<3, BUCKET, FAST>(a, st); break;
    }
}

// T_min frames (raster records) project with the approximate arithmetic,
// reference-compatible frames with the exact one, in both orderings.
void launch_frame_project(const FrameArgs& a, int deg, cudaStream_t st, bool bucket)
{
    if (a.num_tiles == 0) return;
    const bool fast = a.raster_mode != 0;
    if (bucket && fast)
        launch_frame_mode<true, true>(a, deg, st);
    else if (bucket)
        launch_frame_mode<true, false>(a, deg, st);
    else if (fast)
        launch_frame_mode<false, true>(a, deg, st);
    else
        launch_frame_mode<false, false>(a, deg, st);
}

void launch_large_overlaps(const FrameArgs& a, int num_sms, cudaStream_t st)
{
    launch_frame_step(large_overlap_kernel, (unsigned)(num_sms * 4), 256, 0, st, true, a);
}

void launch_count_stage(const FrameArgs& a, cudaStream_t st)
{
    const unsigned grid = (unsigned)a.num_tiles;
    if (grid == 0) return;
    count_stage_kernel<<<grid, 256, 0, st>>>(a);
}

void launch_view_base(const int64_t* view_total, int num_views, int64_t* view_base, int64_t* total, cudaStream_t st)
{
    view_base_kernel<<<1, 32, 0, st>>>(view_total, num_views, view_base, total);
}

void launch_emit(const EmitArgs& a, cudaStream_t st)
{
    const int64_t items = (int64_t)a.num_views * a.n;
    const unsigned grid = (unsigned)((items + 255) / 256);
    if (grid == 0) return;
    emit_kernel<<<grid, 256, 0, st>>>(a);
}

}  // namespace gs
