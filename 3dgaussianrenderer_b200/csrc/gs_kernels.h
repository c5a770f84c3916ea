// Kernel argument blocks and launchers of the gs_b200 pipeline (internal).
#pragma once

#include "gs_common.cuh"

#include <atomic>
#include <utility>

namespace gs {

constexpr int kErrTimeout = 4;  // GS_ERR_DEVICE_TIMEOUT

// Runs a set-up step once per device.  Function attributes such as
// cudaFuncAttributeMaxDynamicSharedMemorySize belong to the current
// device's context, so a kernel that needs more than 48 KB of dynamic
// shared memory must be opted in on every device it runs on, not once per
// process.  Devices 0..63 are remembered; higher ones repeat the step on
// every call (it is idempotent).
class PerDeviceOnce {
public:
    template <class F>
    void run(F&& f)
    {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess) {
            cudaGetLastError();
            dev = -1;
        }
        if (dev < 0 || dev >= 64) {
            f();
            return;
        }
        const uint64_t bit = 1ull << dev;
        if (done_.load(std::memory_order_acquire) & bit) return;
        f();
        done_.fetch_or(bit, std::memory_order_acq_rel);
    }

private:
    std::atomic<uint64_t> done_{0};
};

// Multiprocessor count of the current device (queried once per device).
inline int device_sm_count()
{
    static std::atomic<int> cache[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return 148;
    }
    if (dev >= 0 && dev < 64) {
        const int c = cache[dev].load(std::memory_order_relaxed);
        if (c > 0) return c;
    }
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) {
        cudaGetLastError();
        return 148;
    }
    if (dev >= 0 && dev < 64) cache[dev].store(sms, std::memory_order_relaxed);
    return sms;
}

// What the host learns of a bucket frame, in pinned memory that the kernels
// write: the emission the counts, and the times (globaltimer, ns) the kernels
// at the stages' ends.  Events between the stages, whose records a graph runs
// as nodes of their own, cost a frame 22 us of wall time.
enum FrameTime { kTimeStart, kTimeEmit, kTimeSort, kTimeRaster, kTimeEnd, kFrameTimes };
struct FrameResult {
    unsigned long long t[kFrameTimes];
    int64_t total;             // K
    unsigned long long slots;  // slots (low 32 bits) and overlap chunks (high)
    unsigned long long units;  // units of large splats
    int err;
    int overflow;
};

__device__ __forceinline__ void stamp(FrameResult* r, const FrameTime k)
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    r->t[k] = t;
}

// The kernels of a bucket frame follow one another on the stream with
// programmatic dependent launch: a kernel's blocks are scheduled while the one
// before finishes its last ones, and wait in frame_step_begin until it has
// completed and its writes are visible (single view of 100k Gaussians 159 ->
// 152 us, of 1M 305 -> 295 us; batches unchanged).  Every block of every such kernel waits,
// so a kernel's completion implies that of all before it.  The first loads after
// the wait whose address does not come from another such load are plain ones:
// a read-only load (__ldg) may be moved up across the wait.
__device__ __forceinline__ void frame_step_begin()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... Params, class... Args>
void launch_frame_step(void (*kernel)(Params...), const unsigned grid, const unsigned block, const size_t smem,
                       cudaStream_t st, const bool overlap, Args&&... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = overlap ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);  // errors: the caller's cudaGetLastError
}

// Splats of more than kLargeCandidates candidate tiles are walked by
// large_overlap_kernel, kUnitCandidates at a time (a threshold of 64 takes 7.2
// instead of 8.0 ms for both kernels on the 4K view of 10M large splats, but
// costs the warp walk the register that keeps its ballots: 0.4 ms on 64 views
// of 3M).
constexpr int kLargeCandidates = 32;
constexpr int kUnitCandidates = 1024;

// Fused SH + projection + count + scan over (view, Gaussian) pairs.  A block
// owns one group of 256 Gaussians for `views_per_block` consecutive views;
// every view has its own look-back chain over the groups, so offsets are
// relative to the view's first key.
struct FrameArgs {
    int64_t n;          // Gaussians per view
    int64_t groups;     // ceil(n / 256)
    int32_t num_views;
    int32_t views_per_block;
    uint32_t epoch;     // look-back epoch of this launch
    const uint32_t* epoch_dev;  // non-null: the epoch is read here (graph replays)
    int64_t num_tiles;  // blocks = ceil(num_views / views_per_block) * groups
    const float4* pos;
    const float4* sr;
    const float* sh;    // grouped [ceil(n/256)][sh_count][256]
    int32_t sh_count;
    const float4* color_in;  // degree-0 scenes: colour from the model
    const ViewParams* views;
    const int32_t* orig;  // caller index of each stored Gaussian (null: stored in caller order)
    // outputs, per view at [view * n + i]; offsets for every Gaussian, the
    // rest only for Gaussians that overlap at least one tile
    int32_t raster_mode;  // GS_TERM_REFERENCE: color/xy/conic; GS_TERM_TMIN: rec
    float4* color;
    float2* xy;         // reference mode, or any mode when the rectangle has > 32 candidates
    float* z;
    float4* ell;        // only when the rectangle has > 32 candidates (buckets: > kLargeCandidates, also rect)
    float4* conic;
    float4* rec;        // GS_TERM_TMIN raster record, 3 float4 per item (RasterRec)
    int2* rect;
    uint32_t* hitmask;  // bit c = candidate c overlaps (rectangles with <= 32 candidates)
    int32_t* offsets;   // exclusive key offset inside the view
    // scratch
    uint64_t* status;   // [num_views][groups] look-back words
    unsigned long long* tile_counter;
    int64_t* view_total;  // [num_views] keys per view
    int* err;
    // tile-bucket pipeline (launch_frame_project with bucket = true): the
    // (view, Gaussian) pairs with candidate tiles take slots in any order;
    // every per-item output above is written at the slot instead of
    // view * n + i, `offsets[slot]` receives view * n + caller index,
    // `depth[slot]` the key's depth bits; tile_count[view tile offset + tile]
    // counts the tile's keys and each overlap is recorded in the overlap list.
    uint32_t* depth;
    uint32_t* tile_count;
    unsigned long long* slot_counter;  // slots (low 32 bits) and overlap chunks (high) taken
    uint2* overlaps;                   // [32 * chunk_capacity], see BucketEmitArgs
    uint4* chunks;                     // [chunk_capacity]
    int64_t chunk_capacity;
    FrameResult* result;               // out: the frame's start
    unsigned int* zero_words;          // [zero_count] cleared for the kernels that follow
    int32_t zero_count;
    // splats of more than kLargeCandidates candidate tiles, in units
    uint2* units;                      // [unit_capacity] (slot, unit of the splat)
    unsigned long long* unit_count;    // units listed
    unsigned long long* unit_counter;  // units handed out; zero at launch
    int64_t unit_capacity;
    // probe outputs (diagnostics and tests; null in ordinary frames): the
    // projection of every Gaussian of every view at [view * n + caller
    // index] -- culled Gaussians as centre (-128, -128), depth -128, zero
    // ellipse and conic -- and the colour of those that reach a tile
    float2* probe_xy;
    float* probe_z;
    float4* probe_ell;
    float4* probe_conic;
    float4* probe_color;
};

// The raster order: half-octave classes of the tiles' key counts; the raster's
// launches (host-output frames have several).
constexpr int kOrderClasses = 32;
constexpr int kMaxRasterGroups = 16;

// The overlap list of a tile-bucket frame, in chunks of 32 places.  Chunk c:
//   chunks[c] = (mask of the places that hold an overlap, first slot of the
//                warp that wrote it, its lanes that own a slot, -)
//   overlaps[32 c + j] = (global tile | owner lane << kOverlapTileBits, rank in the tile)
// The slot of an overlap is the first slot + the slot-owning lanes below the
// owner.  A frame whose overlaps need more than chunk_capacity chunks is
// flagged by the tile scan and redone.
constexpr int kOverlapTileBits = 27;

// Bucket emission: every overlap of slot s is written as
// (depth bits << 32 | s) at its rank in its tile's range.
struct BucketEmitArgs {
    const unsigned long long* slot_counter;
    const uint2* overlaps;
    const uint4* chunks;
    int64_t chunk_capacity;
    const uint32_t* depth;           // [slots]
    int32_t* ranges;                 // [2 * tiles]
    int64_t tiles;
    const int* overflow;             // either set: the frame does not stand; all ranges and the big-tile lists
    const int* err;                  // are emptied
    const int64_t* total;
    const unsigned long long* unit_count;
    FrameResult* result;             // out: all but the frame's and the sort's and raster's times
    unsigned int* big_count;
    unsigned int* huge_count;
    int32_t* order;                  // [tiles] out: the raster order; null: not wanted
    int32_t groups;                  // as for the tile scan
    int64_t group_tile[kMaxRasterGroups];
    const unsigned int* class_tiles;
    unsigned int* class_heads;       // [groups * kOrderClasses] placed so far; zero at launch
    uint64_t* keys;
    unsigned long long* batch_counter;  // chunks handed out; zero at launch
};

// Exclusive scan of the per-tile key counts into tile ranges; the last block
// writes the key total.  Ranges are clamped to `capacity` (a frame whose keys do
// not fit is flagged, never overrun).
struct TileScanArgs {
    uint32_t* count;                 // [tiles]; zeroed again after the scan
    int64_t tiles;
    int32_t* ranges;                 // [2 * tiles] out: first, one past last
    uint64_t* status;                // look-back words, one per kTileScanItems tiles
    unsigned long long* block_counter;
    uint32_t epoch;
    const uint32_t* epoch_dev;       // non-null: epoch read here
    int* err;
    int64_t* total;                  // K
    int64_t capacity;
    int* overflow;                   // K > capacity, or another list of the frame was too short
    const unsigned long long* slot_counter;
    int64_t chunk_capacity;
    const unsigned long long* unit_count;  // of the large splats
    int64_t unit_capacity;
    int32_t* big_list;               // out: [0, tiles) tiles with more than fused_cap keys, up to
                                     // kTileSortSmemKeys; [tiles, 2 tiles) the larger ones
    unsigned int* big_count;
    unsigned int* huge_count;
    int32_t fused_cap;
    // raster order: tiles by group (the raster's launches), in each group by class
    int32_t groups;
    int64_t group_tile[kMaxRasterGroups];  // first tile of each group
    unsigned int* class_tiles;       // [groups * kOrderClasses] tiles of each class; zero at launch
    int32_t overlap;                 // 1: follows the large splats' kernel directly
};

// Per-tile sort of the buckets: each tile's keys are ordered by depth and,
// among equal depths, by view * n + i, which is the order of a stable sort
// of the reference's (tile | depth) keys emitted in Gaussian order.
struct TileSortArgs {
    const int32_t* ranges;
    int64_t tiles;
    uint64_t* keys;                  // bucketed (depth << 32 | slot); reordered in place
    uint64_t* keys_alt;              // scratch for tiles above the shared-memory capacity
    int32_t* vals;                   // out: slots in blend order
    int32_t* vals_alt;
    const int32_t* slot_gi;
    int32_t* big_list;               // tiles above the fused capacity (from the tile scan; the
                                     // tiles above kTileSortSmemKeys from index `tiles` on)
    unsigned int* big_count;
    const unsigned int* huge_count;
    int32_t prefix_bits;             // depth bits the radix passes sort (8..32; 0 = 16)
    FrameResult* result;             // out: the sort's start
};
constexpr int kTileSortSmemKeys = 4096;
// Tiles of up to kTileSortHugeMax keys (16-bit counters) are sorted in the
// shared memory of one 1024-thread CTA (tile_sort_huge_kernel), which holds
// kTileSortHugeKeys at a time; larger ones by passes through global memory.
constexpr int kTileSortHugeKeys = 16384;
constexpr int kTileSortHugeMax = 65535;
// Keys a tile may have to be sorted inside its raster CTA (8 per two
// pixels); larger tiles are sorted ahead of the raster.
constexpr int kFusedIpt = 8;
inline int fused_tile_capacity(int tile_w, int tile_h) { return tile_w * tile_h / 2 * kFusedIpt; }
constexpr int kTileScanItems = 1024;  // tiles per scan block

struct EmitArgs {
    int64_t n;
    int32_t num_views;
    const ViewParams* views;
    const int32_t* offsets;
    const int64_t* view_total;
    const int64_t* view_base;  // exclusive prefix of view_total
    const int2* rect;
    const uint32_t* hitmask;  // null: always re-test candidates
    const float2* xy;
    const float4* ell;
    const float* z;
    uint64_t* keys;
    int32_t* values;
    int64_t capacity;
};

// Raster record of one (view, Gaussian) for GS_TERM_TMIN, written by the
// frame kernel: alpha at an offset (dx, dy) from the centre is
// 2^(A dx^2 + B dx dy + C dy^2 + L) -- the conic scaled by -log2(e)/2 and
// L = log2(opacity), so alpha = opacity * exp(-q/2) with one exp2 -- and
// the cull extents bound the ellipse where alpha = kCullAlpha.  A record
// whose conic is not positive definite (non-finite projections) has
// L = -1e30 and empty extents: it contributes nothing, as the reference's
// saturate(NaN) = 0 makes it.
//   r0 = (x, y, ext_x, ext_y)   r1 = (A, B, C, L)   r2 = (red, green, blue, 0)
// (the cull test reads r0 only; r1 and r2 are read for the kept entries)
constexpr float kCullAlpha = 3.814697265625e-06f;  // 2^-18

// Onesweep LSD radix sort of (uint64 key, int32 value) pairs.  Tiles of
// 2048, 4096 or 8192 keys (sort_tile_items(variant)); kSortTile is the
// default variant's, kSortMinTile sizes the look-back words for all.
constexpr int kSortTile = 4096;
constexpr int kSortMinTile = 2048;
constexpr int kSortVariants = 4;
constexpr int kRadix = 256;
constexpr int kMaxPasses = 8;

struct SortScratch {
    uint32_t* hist;                   // [kMaxPasses][kRadix]
    uint64_t* status;                 // [max_tiles][kRadix] look-back words, reused by every pass
    unsigned long long* counters;     // [kMaxPasses] tile counters
    int* err;
    int64_t max_tiles;
};

struct RasterArgs {
    ViewParams view0;                 // the first view, by value (the only one of a single-view launch)
    const ViewParams* views;          // all views
    int32_t num_views;
    int32_t write_empty;              // 1: tiles without entries are written as (0,0,0,0)
    int64_t num_tiles_total;          // sum of the views' tiles (of this launch's tiles when tile_base is used)
    int64_t tile_base;                // CTA b draws global tile order[tile_base + b], or tile_base + b
    const int32_t* ranges;            // [2 * num_tiles_total]
    const int32_t* values;
    const float2* xy;                 // indexed by value (reference-mode kernel)
    const float4* conic;
    const float4* color;
    const float4* rec;                // 3 float4 per value (record kernel); null: use xy/conic/color
    float t_min;
    unsigned long long* tile_counter; // persistent record raster only
    // tile-bucket frames: a tile of at most fused_cap keys is sorted by its
    // raster CTA from the bucketed (depth << 32 | slot) keys; `values` then
    // only holds the order of the larger tiles.  keys == null: `values`
    // holds every tile's order.
    const uint64_t* keys;
    const int32_t* slot_gi;
    int32_t fused_cap;
    const int32_t* order;             // the raster order of the tiles; null: as numbered
    FrameResult* result;              // out: the raster's times; null: not wanted
    int32_t overlap;                  // 1: follows the sort directly, see launch_frame_step
    int32_t stamp_start;              // 1: the first CTA stamps the raster's start
    int32_t end_ctas;                 // the last so many CTAs stamp its end (and long tiles, stamp_end); 0: none
    // record raster (GS_TERM_TMIN) knobs: entries between two tests of whether
    // a block is done (32 or 64), and a persistent grid over the atomic tile queue
    // (tile_counter, zero at launch) instead of one CTA per tile
    int32_t rec_chunk;
    int32_t rec_persistent;
    int32_t sort_prefix_bits;         // depth bits the fused tile sort radix-sorts (8..32; 0 = 16)
};

void launch_sh_stage(int64_t n, const float4* pos, const float* sh, int sh_count, int deg, const ViewParams& v,
                     float4* color, cudaStream_t st);
void launch_project_stage(int64_t n, const float4* pos, const float4* sr, const ViewParams& v, float2* xy,
                          float* z, float4* ell, float4* conic, cudaStream_t st);
void launch_frame_project(const FrameArgs& a, int deg, cudaStream_t st, bool bucket = false);
void launch_tile_scan(const TileScanArgs& a, cudaStream_t st);
void launch_emit_bucket(const BucketEmitArgs& a, int num_sms, cudaStream_t st);
void launch_tile_sort(const TileSortArgs& a, int num_sms, cudaStream_t st);
void launch_large_overlaps(const FrameArgs& a, int num_sms, cudaStream_t st);
void launch_count_stage(const FrameArgs& a, cudaStream_t st);
// view_base[v] = sum of view_total[u < v]; *total = sum of all.
void launch_view_base(const int64_t* view_total, int num_views, int64_t* view_base, int64_t* total, cudaStream_t st);
void launch_emit(const EmitArgs& a, cudaStream_t st);

// Sorts num_items pairs on bits [0, key_bits).  When d_num_items is non-null
// the item count is read on the device (graph-friendly; num_items is then
// an upper bound used to size the grids); likewise a non-null d_epoch
// replaces `epoch` as the look-back epoch of the first pass.  Returns the
// number of passes; the result is in the alternate buffers when that number
// is odd.
int launch_sort(const uint64_t* keys_in, const int32_t* vals_in, uint64_t* keys_alt, int32_t* vals_alt,
                int64_t num_items, const int64_t* d_num_items, int key_bits, const SortScratch& s, uint32_t epoch,
                int num_sms, cudaStream_t st, int variant = 0, const uint32_t* d_epoch = nullptr);
int sort_tile_items(int variant);
int sort_passes(int key_bits);

void launch_ranges(const uint64_t* keys, int64_t num_items, const int64_t* d_num_items, int32_t* ranges,
                   cudaStream_t st);
void launch_density_probe(int64_t n, const float* q, float* wild, float* tame, float* expf_form, cudaStream_t st);
void launch_raster(const RasterArgs& a, int tile_w, int tile_h, int termination, int num_sms, cudaStream_t st);

// Scene storage order (gs_scene.cu): 30-bit Morton codes of the centres over
// the box [lo, hi] with values = index, then the gather of every scene array
// through the sorted permutation (orig[j] = caller index of stored j).
void launch_morton(int64_t n, const float4* pos, const float lo[3], const float hi[3], uint64_t* keys, int32_t* vals,
                   cudaStream_t st);
void launch_scene_gather(int64_t n, const int32_t* perm, const float4* pos_in, const float4* sr_in,
                         const float4* col_in, const float* sh_in, int32_t sh_count, float4* pos, float4* sr,
                         float4* col, float* sh, int32_t* orig, cudaStream_t st);

}  // namespace gs
