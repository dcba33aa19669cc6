// gs_raster.cu — K3 tile binning + K4 tile rasteriser.
//
// The reference draws one instanced quad per visible splat with fixed-function
// BlendState::ALPHA_BLENDING onto a Rgba8Unorm target cleared to opaque black
// (src/renderer.rs:162-195, 284-308; src/shader/render.wesl:46-56, 75-181).  This file
// restates that per pixel:
//   * K3 walks the depth-sorted splats, counts the 16x16 tiles each one's footprint touches, scans the
//     counts (block scan + decoupled look-back) and emits (tile, value) pairs; a stable radix sort
//     by tile then groups the values per tile with draw order kept inside each tile.  Frames of few
//     splats and tiles skip the scan, the pairs and their sort (raster_direct_kernel).
//   * K4 runs one CTA per tile; each thread owns one or two pixels and walks the tile's splats in
//     draw order (far to near), staged a chunk at a time in shared memory.  For every fragment
//     it evaluates the interpolated quad offset q, the discard test, the alpha of the display
//     mode, and blends with the 8-bit re-quantisation a Rgba8Unorm attachment performs after
//     every fragment: d' = round(d·(1-α) + s·α) in units of 1/255.
// Fragments whose alpha cannot move an 8-bit channel (see splat_r2_bound) lie outside the splat's
// fragment box and are never visited; skipping them leaves every pixel bit-identical.
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "gs_internal.h"

namespace gs {

constexpr uint32_t kBinThreads = 256;
constexpr uint32_t kRasterThreads = 256;
// A warp's pixel block is 8x4 pixels, or 8x8 with two pixels a thread: its pixel centres span 7 x 3 or 7 x 7.
constexpr float kBlockSpanX = 7.0f;

struct RasterLayout {
    Ctrl *ctrl;          // raster control block: owns the area's epoch counter and flag arena
    Ctrl *sort_ctrl;     // tile sort control block
    uint64_t *flags;     // flag arena, first part: scan look-back flags
    uint64_t *sort_flags;  // flag arena, second part: tile-sort look-back flags
    uint32_t arena_words;  // words of the flag arena (both parts)
    gs_splat *splats;    // several models: their splats side by side, capacity max_splats
    uint4 *info;         // per draw rank: tile rectangle, kept-tile mask, pair value
    uint32_t *offsets;   // per draw rank: tile count, then its exclusive scan
    uint2 *pairs;        // (tile, value), capacity max_pairs
    uint2 *ranges;       // per tile [start, end)
    uint32_t *counts;    // per tile pair count
    bool counting;       // the emission counts them (up to kCountTiles tiles)
    uint32_t *blockcounts;  // per emit CTA and tile pair count (counting path)
    uint32_t *order;     // tiles by descending pair count: the rasteriser's launch order (counting path)
    uint2 *sort_alt;     // the tile sort's ping-pong buffer, capacity max_pairs
    uint32_t tiles_x, tiles_y, ntiles, key_bits;
    uint32_t value_bits;  // compact items (see launch_sort_items): bits of a pair value; 0: whole pairs
    uint32_t *items() const { return reinterpret_cast<uint32_t *>(pairs); }
    uint8_t *low(uint32_t max_pairs) const { return reinterpret_cast<uint8_t *>(pairs) + (size_t)max_pairs * 4; }
};

// Up to kCountTiles tiles (1080p has 8160), the emit kernel counts pairs per tile in shared
// memory; the per-tile counts give the tile-sort histograms and, scanned, the tile ranges.
// Larger targets count per digit instead, and the tile sort's second pass counts per tile.
constexpr uint32_t kCountTiles = 8192;
constexpr uint32_t kEmitBlocks = 152 * 8;

// Ranks a direct frame can have: a bit each in shared memory (RasterShared::raw).
constexpr uint32_t kDirectMaxRanks = 3u * 16u * kRasterThreads * 8u;

constexpr uint32_t kScanItems = 16;
constexpr uint32_t kScanTile = 256 * kScanItems;

// CTAs of a kernel that the current device holds at once (0 when it cannot be told).
template <class K>
static uint32_t resident_ctas(K kernel, uint32_t threads, size_t smem) {
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, (int)threads, smem) != cudaSuccess)
        return 0;
    return (uint32_t)sms * (uint32_t)per_sm;
}

static uint32_t bits_for(uint32_t v) {
    uint32_t b = 1;
    while (b < 32 && (v >> b) != 0) ++b;
    return b;
}

// Scan flags: one per 4096-count tile (plus one), padded to 256 bytes so the tile-sort flags
// after them stay 256-byte aligned.
static size_t scan_flag_words(uint32_t max_splats) {
    return align_up(((size_t)max_splats + kScanTile - 1) / kScanTile + 1, 32);
}

// Scratch: raster control block | tile-sort control block | flag arena (scan flags, tile-sort
// flags) | buffers.  The two control blocks and the arena's start sit at offsets no call size
// moves; the arena's length and everything after it follow (max_splats, width, height, max_pairs).
static RasterLayout raster_layout(void *scratch, uint32_t max_splats, uint32_t w, uint32_t h,
                                  uint32_t max_pairs) {
    RasterLayout L;
    L.tiles_x = (w + GS_TILE - 1) / GS_TILE;
    L.tiles_y = (h + GS_TILE - 1) / GS_TILE;
    L.ntiles = L.tiles_x * L.tiles_y;
    L.key_bits = bits_for(L.ntiles > 0 ? L.ntiles - 1 : 0);
    uint8_t *p = reinterpret_cast<uint8_t *>(scratch);
    L.ctrl = reinterpret_cast<Ctrl *>(p);
    p += align_up(sizeof(Ctrl), 256);
    L.sort_ctrl = reinterpret_cast<Ctrl *>(p);
    p += align_up(sizeof(Ctrl), 256);
    const size_t scan_words = scan_flag_words(max_splats);
    const size_t arena = scan_words + sort_pairs_flag_words(max_pairs, L.key_bits);
    L.flags = reinterpret_cast<uint64_t *>(p);
    L.sort_flags = L.flags + scan_words;
    L.arena_words = (uint32_t)arena;
    p += align_up(arena * sizeof(uint64_t), 256);
    L.splats = reinterpret_cast<gs_splat *>(p);
    p += align_up((size_t)max_splats * sizeof(gs_splat), 256);
    L.info = reinterpret_cast<uint4 *>(p);
    p += align_up((size_t)max_splats * 16, 256);
    L.offsets = reinterpret_cast<uint32_t *>(p);
    p += align_up((size_t)max_splats * 4 + 16, 256);
    L.pairs = reinterpret_cast<uint2 *>(p);
    p += align_up((size_t)max_pairs * 8, 256);
    L.ranges = reinterpret_cast<uint2 *>(p);
    p += align_up((size_t)L.ntiles * sizeof(uint2), 256);
    L.counts = reinterpret_cast<uint32_t *>(p);
    p += align_up((size_t)L.ntiles * 4, 256);
    L.counting = L.ntiles <= kCountTiles;
    L.blockcounts = L.order = nullptr;
    if (L.counting) {
        L.order = reinterpret_cast<uint32_t *>(p);
        p += align_up((size_t)L.ntiles * 4, 256);
        L.blockcounts = reinterpret_cast<uint32_t *>(p);
        p += align_up((size_t)kEmitBlocks * L.ntiles * 4, 256);
    }
    L.sort_alt = reinterpret_cast<uint2 *>(p);
    // Up to 65,536 tiles take two digits, whose high one leaves 24 bits or more for a value.
    const uint32_t bits = bits_for(max_splats);
    L.value_bits = L.key_bits <= 16 && bits < 32 && tile_split(L.key_bits).bits[1] + bits <= 32 ? bits : 0u;
    return L;
}

size_t raster_scratch_bytes(uint32_t max_splats, uint32_t w, uint32_t h, uint32_t max_pairs) {
    const uint32_t tiles = ((w + GS_TILE - 1) / GS_TILE) * ((h + GS_TILE - 1) / GS_TILE);
    const uint32_t key_bits = bits_for(tiles > 0 ? tiles - 1 : 0);
    const size_t arena = scan_flag_words(max_splats) + sort_pairs_flag_words(max_pairs, key_bits);
    return 2 * align_up(sizeof(Ctrl), 256) + align_up(arena * sizeof(uint64_t), 256) +
           align_up((size_t)max_splats * sizeof(gs_splat), 256) + align_up((size_t)max_splats * 16, 256) +
           align_up((size_t)max_splats * 4 + 16, 256) + align_up((size_t)max_pairs * 8, 256) +
           align_up((size_t)tiles * sizeof(uint2), 256) + align_up((size_t)tiles * 4, 256) +
           (tiles <= kCountTiles ? align_up((size_t)tiles * 4, 256) + align_up((size_t)kEmitBlocks * tiles * 4, 256)
                                 : 0) +
           align_up((size_t)max_pairs * 8, 256);
}

const Ctrl *raster_ctrl(const void *scratch) { return reinterpret_cast<const Ctrl *>(scratch); }

Tuning default_tuning() {
    Tuning t;
    if (const char *v = getenv("GS300_SUFFIX_MIN")) t.suffix_min = (uint32_t)strtoul(v, nullptr, 10);
    if (const char *v = getenv("GS300_SUFFIX_EPS")) t.eps = strtof(v, nullptr);
    if (const char *v = getenv("GS300_SORT_DIGIT_BITS")) t.sort_digit_bits = (uint32_t)strtoul(v, nullptr, 10);
    if (const char *v = getenv("GS300_HIST_BLOCKS")) t.hist_blocks = (uint32_t)strtoul(v, nullptr, 10);
    if (const char *v = getenv("GS300_SORT_MATCH")) t.sort_match = (uint32_t)strtoul(v, nullptr, 10) ? 1u : 0u;
    return t;
}

// A tile rectangle in one word: bytes x0, y0, 127 - x1, 127 - y1 of its first and last tile, in units of
// 2^shift tiles so that a target has at most 128 of them each way.  With a tile's own bytes (x, y,
// 127 - x, 127 - y), each below 128, the rectangle can hold the tile when no byte of the difference
// borrows: one subtraction under guard bits.  (With shift 0 it does hold it.)
constexpr uint32_t kRectGuard = 0x80808080u, kEmptyRect = 0x7F7F7F7Fu;
__device__ __forceinline__ uint32_t pack_rect(uint32_t x0, uint32_t y0, uint32_t x1, uint32_t y1, uint32_t shift) {
    return (x0 >> shift) | ((y0 >> shift) << 8) | ((127u - (x1 >> shift)) << 16) | ((127u - (y1 >> shift)) << 24);
}
__device__ __forceinline__ bool rect_may_hold(uint32_t rect, uint32_t tile) {
    return (((tile | kRectGuard) - rect) & kRectGuard) == kRectGuard;
}

// Range of a splat's colour and alpha.  The preprocess writes colours of 0..255 and alphas of 0..1: class 0.
// A caller's own splats may hold others: class k, 1..kColourClasses, for colours within +-255 2^k, whose
// blends stay within them too as long as the alpha is in 0..1; kWildColours for the rest and NaN.
constexpr uint32_t kColourClasses = 12, kWildColours = 15;
__device__ __noinline__ uint32_t colour_class_beyond(float r, float g, float b, float alpha) {
    const float reach = fmaxf(fabsf(r), fmaxf(fabsf(g), fabsf(b))), sum = (r + g) + b;  // the sum is for NaN
    if (!(alpha >= 0.0f && alpha <= 1.0f) || sum != sum || !(reach <= 255.0f * (float)(1u << kColourClasses)))
        return kWildColours;
    uint32_t k = 1;
    while (255.0f * (float)(1u << k) < reach) ++k;
    return k;
}
__device__ __forceinline__ uint32_t colour_class(const float4 c) {
    // as words, floats from 0 on are in order, and below those with a sign and NaN
    const uint32_t most = max(__float_as_uint(c.x), max(__float_as_uint(c.y), __float_as_uint(c.z)));
    const bool in = most <= __float_as_uint(255.0f) && __float_as_uint(c.w) <= __float_as_uint(1.0f);
    return in ? 0u : colour_class_beyond(c.x, c.y, c.z, c.w);
}

// K3a: per draw rank, the splat's tile rectangle, the corner tiles its footprint misses, and
// its tile count.  With `binfo` (the preprocess having stored each visible splat's tiles) the rank
// gathers that 16-byte record; otherwise it gathers the 48-byte splat and works the tiles out here.
// The pair value is the splat's index from `base` on (several models: in their common array.  Four models of
// 6M splats: 174 us a binning with the splats copied into draw order, 70 us with them side by side).
// The first segment's launch (arena non-null) also clears the flag-arena words the call must
// clear, before the scan and the tile sort read any flag.
// DIRECT: the ranks are scanned by raster_direct_kernel up to the capacity: each gets its rectangle in one
// word (`rects`, in place of the count), an empty one where there is no splat or no tile is kept; the first
// segment's launch (reset) starts the call's control block.
// The largest colour_class of `foreign` splats goes to the owner, for direct frames with the pairs to the frame's
// set of sums.
// Bound by the latency of the gather: six CTAs an SM (40 registers) take 249 us a binning of four models of
// 6M splats, five (45 registers) 255.
template <bool DIRECT>
__global__ void __launch_bounds__(kBinThreads, 6) bin_count_kernel(
    const gs_splat *splats, const uint4 *binfo, const uint32_t *sorted_index,
    const uint32_t *count, uint32_t max_count, uint32_t base, int several, int foreign,
    uint32_t tiles_x, uint32_t tiles_y, uint32_t mode, float std2, uint4 *info,
    uint32_t *counts, Ctrl *owner, uint64_t *arena, uint32_t *rects,
    uint32_t rect_shift, int reset, uint32_t arena_words) {
    frame_kernel_enter();
    if (arena) arena_clear(owner, arena);
    const uint32_t set = DIRECT ? owner->direct_next : 0u;
    if (DIRECT && reset && blockIdx.x == 0 && threadIdx.x == 0) {
        ctrl_reset_flagless(owner, arena_words);
        owner->direct_now = set;
    }
    const uint32_t n = count ? min(*count, max_count) : max_count;
    const uint32_t k = blockIdx.x * kBinThreads + threadIdx.x;
    uint4 t = make_uint4(0u, 0u, 0u, 0u);  // x0 | y0 << 16, w | h << 16, mask, count
    uint32_t colours = 0;
    if (k < n) {
        // Indices come from the depth sort; the bound check only matters if that sort timed out.
        const uint32_t gi = sorted_index[k];
        if (gi < max_count) {
            if (binfo) {
                t = binfo[gi];
            } else {
                // all three 16-byte parts in one round trip (the colour bounds the corner-tile test)
                const float4 *src = reinterpret_cast<const float4 *>(splats + gi);
                const float4 a = src[0], q = src[1], c = src[2];
                // ahead of the tile test: the branch keeps the three loads together (8 views of 6M splats 10.96 ms a
                // batch with the class found behind the test, 10.78 so)
                if (foreign) colours = colour_class(c);
                t = splat_tile_info(a, q, c, tiles_x, tiles_y, mode, std2);
                if (t.w == 0u) colours = 0u;
            }
        }
        info[k] = make_uint4(t.x, t.y, t.z, base + gi);
    }
    if constexpr (DIRECT) {
        if (k < max_count)
            rects[k] = t.w ? pack_rect(t.x & 0xFFFFu, t.x >> 16, (t.x & 0xFFFFu) + (t.y & 0xFFFFu) - 1u,
                                       (t.x >> 16) + (t.y >> 16) - 1u, rect_shift)
                           : kEmptyRect;
        if (colours) atomicMax(&owner->direct_class[set], colours);
        const uint32_t pairs = __reduce_add_sync(0xFFFFFFFFu, t.w);
        if ((threadIdx.x & 31u) == 0 && pairs) atomicAdd(&owner->direct_pairs[set], pairs);
    } else {
        if (k < n) counts[k] = t.w;
        else if (k < max_count && several) counts[k] = 0u;  // the scan covers every segment's capacity
        if (colours) atomicMax(&owner->colours, colours);
    }
}

// K3b: exclusive scan of the tile counts in place (decoupled look-back over 4096-count tiles);
// the last tile records the pairs wanted and kept, and a list overflow.
__global__ void __launch_bounds__(256) bin_scan_kernel(uint32_t *data, const uint32_t *count,
                                                       uint32_t max_count, uint32_t max_pairs, Ctrl *ctrl,
                                                       uint64_t *flags) {
    __shared__ uint32_t s_warp[8];
    __shared__ uint32_t s_tile, s_epoch, s_prefix, s_limit, s_stall;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    frame_kernel_enter();
    if (tid == 0) {
        s_epoch = *(volatile uint32_t *)&ctrl->epoch;
        s_limit = ctrl->spin_limit;
        s_stall = ctrl->stall_tile;
        s_tile = blockIdx.x;  // look-back predecessors are lower, earlier-dispatched CTAs
    }
    __syncthreads();
    const uint32_t n = count ? min(*count, max_count) : max_count;
    const uint32_t ntiles = (n + kScanTile - 1) / kScanTile;
    const uint32_t tile = s_tile, epoch = s_epoch;
    if (tile >= ntiles) return;
    const uint32_t base = tile * kScanTile + tid * kScanItems;
    uint32_t v[kScanItems];
    if (base + kScanItems <= n) {
#pragma unroll
        for (uint32_t i = 0; i < kScanItems; i += 4) {
            const uint4 x = *reinterpret_cast<const uint4 *>(data + base + i);
            v[i] = x.x;
            v[i + 1] = x.y;
            v[i + 2] = x.z;
            v[i + 3] = x.w;
        }
    } else {
#pragma unroll
        for (uint32_t i = 0; i < kScanItems; ++i) v[i] = base + i < n ? data[base + i] : 0u;
    }
    uint32_t sum = 0;
#pragma unroll
    for (uint32_t i = 0; i < kScanItems; ++i) sum += v[i];
    uint32_t x = sum;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t wv = lane < 8 ? s_warp[lane] : 0u;
        uint32_t wi = wv;
#pragma unroll
        for (uint32_t o = 1; o < 8; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, wi, o);
            if (lane >= o) wi += y;
        }
        const uint32_t total = __shfl_sync(0xFFFFFFFFu, wi, 7);
        if (lane == 0)
            publish_flag(flags + tile, tile, s_stall, pack_flag(epoch, tile == 0 ? kFlagPrefix : kFlagAggregate, total));
        const uint32_t prefix = tile == 0 ? 0u : look_back_warp(flags, tile, epoch, &ctrl->status, s_limit);
        if (lane < 8) s_warp[lane] = wi - wv;  // exclusive per-warp offsets
        if (lane == 0) {
            const uint64_t incl = (uint64_t)prefix + total;
            const uint32_t sat = incl > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)incl;
            if (tile > 0) publish_flag(flags + tile, tile, s_stall, pack_flag(epoch, kFlagPrefix, sat));
            s_prefix = prefix;
            if (tile == ntiles - 1) {
                ctrl->total = sat;
                ctrl->count = min(sat, max_pairs);
                if (sat > max_pairs) atomicOr(&ctrl->status, kStatusCapacity);
            }
        }
    }
    __syncthreads();
    uint32_t run = s_prefix + s_warp[warp] + x - sum;
    if (base + kScanItems <= n) {
#pragma unroll
        for (uint32_t i = 0; i < kScanItems; i += 4) {
            uint4 o;
            o.x = run;
            run += v[i];
            o.y = run;
            run += v[i + 1];
            o.z = run;
            run += v[i + 2];
            o.w = run;
            run += v[i + 3];
            *reinterpret_cast<uint4 *>(data + base + i) = o;
        }
    } else {
#pragma unroll
        for (uint32_t i = 0; i < kScanItems; ++i) {
            if (base + i < n) data[base + i] = run;
            run += v[i];
        }
    }
}

// Place, in its w x h rectangle, of the n-th kept tile of a splat (n < its tile count).  The
// kept-tile mask (splat_tile_info) only ever drops corner tiles, at places 0, w-1, (h-1)w and
// hw-1, so the place is n moved past each dropped corner at or before it, in increasing order
// (the last corner has no place after it): cheaper than a general n-th-set-bit search.
__device__ __forceinline__ uint32_t kept_tile_place(uint32_t m, uint32_t w, uint32_t h, uint32_t n) {
    uint32_t pos = n;
    if (!(m & 1u)) ++pos;
    if (w > 1u && !((m >> (w - 1u)) & 1u) && pos >= w - 1u) ++pos;
    const uint32_t c2 = (h - 1u) * w;
    if (h > 1u && !((m >> c2) & 1u) && pos >= c2) ++pos;
    return pos;
}

// K3c: every splat writes its (tile, value) pairs at its scanned offset, its kept tiles in
// row-major order.  A warp takes an equal share of the pairs, not of the ranks: the nearest splats of
// a close-up cover thousands of tiles each and lie next to one another in draw order (400k splats at
// 1366x768 from inside the scene: 97 us by ranks, 16 by pairs).  It finds its first rank by a 32-way
// search of the offsets, then goes through windows of 32 ranks: pair r of a window goes to lane r mod
// 32, which finds its splat among the window's in shared memory and its tile from the pair's place in
// the splat's rectangle (its kept tiles skip the dropped corners).  Stores are consecutive.  Bound by
// issue: 24.7M pairs took 136 us with the splat found by a binary search of shuffles and its fields by
// seven more, 126 with an or-reduction and three shared loads; five CTAs an SM, as six (40 registers)
// spill time into the digit counts of large targets (3M / 4K: 226 us a binning, 237).
// Also accumulates the tile counts (or the tile-key digit histograms of the tile sort) in
// shared memory; each CTA hands its shared bins on once.
// COUNTS: one counter per tile, else the digit histograms; COMPACT: items and low digits, else pairs.
constexpr uint32_t kEmitMin = 96;  // pairs of a warp's share at least (its search costs about 3 us)

// A warp's window of 32 ranks.
struct EmitWindow {
    uint4 rect[32], at[32];
    uint8_t nth[32];
};

template <bool COUNTS, bool COMPACT>
__global__ void __launch_bounds__(kBinThreads, 5) bin_emit_kernel(
    const uint4 *info, const uint32_t *offsets, const uint32_t *count, uint32_t max_count,
    uint2 *pairs, uint32_t max_pairs, uint32_t value_bits, uint32_t tiles_x, uint32_t ntiles, Ctrl *ctrl,
    Ctrl *sort_ctrl, const PassSplit split, uint32_t *blockcounts) {
    extern __shared__ uint32_t s_bins[];
    __shared__ EmitWindow s_win[kBinThreads / 32];
    const uint32_t nbins = COUNTS ? ntiles : 4u * 256u;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, lt = lanemask_lt(), le = lt | (1u << lane);
    EmitWindow &win = s_win[tid >> 5];
    for (uint32_t i = tid; i < nbins; i += kBinThreads) s_bins[i] = 0u;
    frame_kernel_enter();
    const uint32_t n = count ? min(*count, max_count) : max_count;
    const uint32_t total = ctrl->total;
    // a scan that gave up leaves offsets nothing can be found by (status already set): emit nothing
    const bool sound = !(*(volatile uint32_t *)&ctrl->status & kStatusTimeout);
    __syncthreads();
    uint32_t *items = reinterpret_cast<uint32_t *>(pairs);
    uint8_t *low = reinterpret_cast<uint8_t *>(pairs) + (size_t)max_pairs * 4u;
    const uint32_t low_bits = split.bits[0], low_mask = (1u << low_bits) - 1u;
    auto emit = [&](uint32_t t, uint32_t value, uint32_t at) {
        if (at < max_pairs) {
            if constexpr (COMPACT) {
                items[at] = ((t >> low_bits) << value_bits) | value;
                low[at] = (uint8_t)(t & low_mask);
            } else {
                pairs[at] = make_uint2(t, value);
            }
            if constexpr (COUNTS) {
                if (t < ntiles) atomicAdd(&s_bins[t], 1u);
                else atomicOr(&ctrl->status, kStatusBounds);
            } else {
                for (uint32_t p = 0; p < split.n; ++p)
                    atomicAdd(&s_bins[p * 256u + ((t >> split.shift[p]) & ((1u << split.bits[p]) - 1u))], 1u);
            }
        }
    };
    const uint32_t warps = gridDim.x * (kBinThreads / 32u), w = blockIdx.x * (kBinThreads / 32u) + (tid >> 5);
    const uint32_t share = max(kEmitMin, (uint32_t)(((uint64_t)total + warps - 1u) / warps));
    const uint64_t first = (uint64_t)w * share;
    if (sound && n > 0 && first < total) {
        const uint32_t q0 = (uint32_t)first, q1 = (uint32_t)min((uint64_t)total, first + share);
        // the last rank from lo on whose offset is at or before q (offsets[lo] is): the one that holds
        // pair q, as ranks without pairs share the next one's offset
        auto rank_of = [&](uint32_t q, uint32_t lo) {
            uint32_t hi = n;
            while (hi - lo > 1u) {
                const uint32_t step = (hi - lo + 31u) / 32u, at = lo + lane * step;
                const uint32_t m = __ballot_sync(0xFFFFFFFFu, at < hi && offsets[at] <= q);
                lo += (m ? 31u - __clz(m) : 0u) * step;
                hi = min(hi, lo + step);
            }
            return lo;
        };
        uint32_t empty = 0;  // windows without pairs in a row
        for (uint32_t k0 = rank_of(q0, 0); k0 < n; k0 += 32u) {
            const uint32_t k = k0 + lane;
            uint4 in = make_uint4(0u, 0u, 0u, 0u);
            uint32_t from = q1, to = q1, off = q1;  // this rank's pairs of the warp's share
            if (k < n) {
                in = info[k];
                off = offsets[k];
                const uint32_t next = (k + 1 < n) ? offsets[k + 1] : total;
                // A count beyond the splat's tile rectangle can only come from a bad scan: emit nothing for it.
                if (next >= off && next - off <= (in.y & 0xFFFFu) * (in.y >> 16)) {
                    from = min(max(off, q0), q1);
                    to = min(max(next, q0), q1);
                } else {
                    atomicOr(&ctrl->status, kStatusBounds);
                }
            }
            const bool more = __shfl_sync(0xFFFFFFFFu, to, 31) < q1;
            const uint32_t cnt = to - from;
            // warp-exclusive prefix of the counts: this lane's pairs are [excl, excl + cnt) of the run
            uint32_t incl = cnt;
#pragma unroll
            for (uint32_t d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, d);
                if (lane >= d) incl += y;
            }
            const uint32_t excl = incl - cnt, run = __shfl_sync(0xFFFFFFFFu, incl, 31);
            // The window's splats in shared memory, and its lanes that have pairs in order: pair r of the
            // run belongs to the last of them that starts at or before r, which a round counts with one
            // or-reduction of its 32 places' starts.
            const uint32_t iw = in.y & 0xFFFFu;
            const uint32_t some = __ballot_sync(0xFFFFFFFFu, cnt != 0u);
            __syncwarp();
            win.rect[lane] = in;  // x0 | y0 << 16, w | h << 16, kept-tile mask, value
            win.at[lane] = make_uint4(from - excl, off, __float_as_uint(iw ? 1.0f / (float)iw : 0.0f), 0u);
            if (cnt) win.nth[__popc(some & lt)] = (uint8_t)lane;
            __syncwarp();
            uint32_t before = 0;  // lanes of `some` that start ahead of the round
            for (uint32_t r0 = 0; r0 < run; r0 += 32) {
                const uint32_t r = r0 + lane, place = excl - r0;
                const uint32_t starts = __reduce_or_sync(0xFFFFFFFFu, cnt && place < 32u ? 1u << place : 0u);
                const uint32_t src = win.nth[before + __popc(starts & le) - 1u];
                before += __popc(starts);
                if (r < run) {
                    const uint4 rc = win.rect[src], ra = win.at[src];
                    const uint32_t sw = rc.y & 0xFFFFu, at = ra.x + r, local = at - ra.y;  // place among its kept tiles
                    // rc.z: tiles kept of a rectangle of at most 16 (bit ty·w + tx); 0 = all of it
                    const uint32_t pos = rc.z ? kept_tile_place(rc.z, sw, rc.y >> 16, local) : local;
                    // row = floor(pos / w), exact in float: pos < 2^24 and the error of 1/w is
                    // far below the 1/w gap between pos/w and the next integer
                    const uint32_t ty = (uint32_t)(((float)pos + 0.5f) * __uint_as_float(ra.z)), tx = pos - ty * sw;
                    emit(((rc.x >> 16) + ty) * tiles_x + (rc.x & 0xFFFFu) + tx, rc.w, at);
                }
            }
            if (!more) break;
            // a long stretch of ranks without pairs (another model's unused capacity, splats outside the
            // target) is passed over by another search
            empty = run ? 0u : empty + 1u;
            if (empty == 4u) {
                empty = 0;
                const uint32_t here = __shfl_sync(0xFFFFFFFFu, to, 31), at = k0 + 31u;
                k0 = max(k0, rank_of(here, at) - 32u);  // at + 1 <= the rank found, or no rank is left
            }
        }
    }
    __syncthreads();
    if constexpr (COUNTS) {
        // every CTA of the grid writes its slice (zeros when it had no pairs): plain stores,
        // summed per tile by tile_count_kernel
        uint32_t *dst = blockcounts + (size_t)blockIdx.x * ntiles;
        for (uint32_t t = tid; t < ntiles; t += kBinThreads) dst[t] = s_bins[t];
    } else {
        for (uint32_t p = 0; p < split.n; ++p) {
            const uint32_t v = s_bins[p * 256u + tid];
            if (v) atomicAdd(&sort_ctrl->hist[p][tid], v);
        }
        // the last CTA to finish turns the digit histograms into exclusive offsets, a warp a pass
        __shared__ uint32_t s_last;
        __threadfence();
        __syncthreads();
        if (tid == 0) s_last = atomicAdd(&sort_ctrl->ticket[7], 1u) == gridDim.x - 1u ? 1u : 0u;
        __syncthreads();
        const uint32_t p = tid >> 5;
        if (s_last && p < split.n) {
            __threadfence();
            uint32_t v[8], sum = 0;
#pragma unroll
            for (uint32_t j = 0; j < 8; ++j) sum += v[j] = __ldcg(&sort_ctrl->hist[p][lane * 8u + j]);
            uint32_t run = sum;
#pragma unroll
            for (uint32_t d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, run, d);
                if (lane >= d) run += y;
            }
            run -= sum;
#pragma unroll
            for (uint32_t j = 0; j < 8; ++j) {
                sort_ctrl->hist[p][lane * 8u + j] = run;
                run += v[j];
            }
        }
    }
}

// [start, end) of every tile from its pair count where the target has too many tiles for
// tile_scan_kernel: one CTA, 8192 tiles at a time (4K: 4 rounds, 17 us; 52 us finding the ends in the
// sorted pairs).
__global__ void __launch_bounds__(1024) tile_starts_kernel(const uint32_t *counts, uint32_t ntiles,
                                                           uint2 *ranges) {
    __shared__ __align__(16) uint32_t s_v[8192 + 4];
    __shared__ uint32_t s_w[32];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    frame_kernel_enter();
    uint32_t before = 0;
    for (uint32_t t0 = 0; t0 < ntiles; t0 += 8192u) {
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            const uint32_t t = tid + 1024u * j;
            s_v[t] = t0 + t < ntiles ? counts[t0 + t] : 0u;
        }
        __syncthreads();
        uint4 a = *reinterpret_cast<const uint4 *>(&s_v[8u * tid]), b = *reinterpret_cast<const uint4 *>(&s_v[8u * tid + 4u]);
        const uint32_t sum = ((a.x + a.y) + (a.z + a.w)) + ((b.x + b.y) + (b.z + b.w));
        uint32_t inc = sum;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
            if (lane >= o) inc += x;
        }
        if (lane == 31) s_w[warp] = inc;
        __syncthreads();
        uint32_t run = before + inc - sum, all = 0;
        for (uint32_t w = 0; w < 32; ++w) {
            const uint32_t x = s_w[w];
            if (w < warp) run += x;
            all += x;
        }
        const uint32_t c[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        uint32_t first[8];
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            first[j] = run;
            run += c[j];
        }
        *reinterpret_cast<uint4 *>(&s_v[8u * tid]) = make_uint4(first[0], first[1], first[2], first[3]);
        *reinterpret_cast<uint4 *>(&s_v[8u * tid + 4u]) = make_uint4(first[4], first[5], first[6], first[7]);
        before += all;
        if (tid == 0) s_v[8192] = before;
        __syncthreads();
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            const uint32_t t = tid + 1024u * j;
            if (t0 + t < ntiles) ranges[t0 + t] = make_uint2(s_v[t], s_v[t + 1]);
        }
        __syncthreads();
    }
}

// Starts a raster call: its control block and the tile sort's (CTA 0), the tile counts cleared by the
// other CTAs.
__global__ void __launch_bounds__(256) raster_init_kernel(Ctrl *ctrl, Ctrl *sort_ctrl, uint32_t arena_words, WaitCfg cfg,
                                                          uint32_t *counts, uint32_t ntiles) {
    frame_kernel_enter();
    if (blockIdx.x == 0) {
        ctrl_reset(ctrl, ctrl, arena_words, cfg);
        ctrl_reset(sort_ctrl, ctrl, kKeepArena, cfg);
        return;
    }
    for (uint32_t t = (blockIdx.x - 1u) * 1024u + threadIdx.x, e = min(ntiles, blockIdx.x * 1024u); t < e; t += 256u) counts[t] = 0u;
}

// Per-tile pair counts of one segment (the sum over the emit CTAs), added to the running
// counts.  blockIdx.y takes a slice of the emit CTAs, so the sum runs wide, not long.
constexpr uint32_t kCountSlices = 16;

__global__ void __launch_bounds__(256) tile_count_kernel(const uint32_t *blockcounts, uint32_t nblocks,
                                                         uint32_t ntiles, uint32_t *counts) {
    frame_kernel_enter();
    const uint32_t t = blockIdx.x * 256u + threadIdx.x;
    if (t >= ntiles) return;
    const uint32_t per = (nblocks + kCountSlices - 1) / kCountSlices;
    const uint32_t b0 = blockIdx.y * per, b1 = min(nblocks, b0 + per);
    uint32_t part[4] = {0, 0, 0, 0};
    uint32_t b = b0;
    for (; b + 4 <= b1; b += 4)
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) part[q] += blockcounts[(size_t)(b + q) * ntiles + t];
    for (; b < b1; ++b) part[0] += blockcounts[(size_t)b * ntiles + t];
    const uint32_t c = (part[0] + part[1]) + (part[2] + part[3]);
    if (c) atomicAdd(&counts[t], c);
}

// Size class of a tile list for the launch order: two classes per power of two, 0 = empty.
constexpr uint32_t kOrderClasses = 66;
__device__ __forceinline__ uint32_t order_class(uint32_t c) {
    if (c == 0) return 0u;
    const uint32_t lg = 31u - __clz(c);
    return 1u + 2u * lg + (lg > 0 ? (c >> (lg - 1u)) & 1u : 0u);
}

// [start, end) of every tile from the per-tile counts (exclusive scan; one CTA, 8 consecutive tiles a
// thread), the tile sort's exclusive digit offsets, and the rasteriser's launch order: tiles by
// descending size class (a counting sort), so the longest lists start first and the grid does not end
// on a few long tiles that started late.  The order inside a class is whatever the shared atomics give;
// it only schedules CTAs, every tile's pixels are the same in any order.
// One SM's load and store slots bound it, so all global traffic is coalesced through shared memory; the
// high digit's offsets are the scan's values at its first tiles, the low digit's counts strided sums, a
// class takes one atomic a warp, and the class starts one warp's scan (10.7 us at 8160 tiles against 14.5
// with strided accesses, an atomic per tile and digit and a serial walk over the classes).
constexpr uint32_t kScanTilesMax = 8192;
static_assert(kCountTiles <= kScanTilesMax, "8 tiles a thread");
__global__ void __launch_bounds__(1024) tile_scan_kernel(const uint32_t *counts, uint32_t ntiles,
                                                         uint2 *ranges, uint32_t *order,
                                                         Ctrl *sort_ctrl, const PassSplit split) {
    __shared__ __align__(16) uint32_t s_v[kScanTilesMax + 4];
    __shared__ uint32_t s_w[32], s_low[1024], s_lw[10], s_cls[96];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, lt = lanemask_lt();
    if (tid < 96u) s_cls[tid] = 0u;
    frame_kernel_enter();
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j) {
        const uint32_t t = tid + 1024u * j;
        s_v[t] = t < ntiles ? counts[t] : 0u;
    }
    __syncthreads();
    const uint32_t base = tid * 8u;
    uint32_t v[8], sum = 0;
#pragma unroll
    for (uint32_t j = 0; j < 8; j += 4) {
        const uint4 x = *reinterpret_cast<const uint4 *>(&s_v[base + j]);
        v[j] = x.x;
        v[j + 1] = x.y;
        v[j + 2] = x.z;
        v[j + 3] = x.w;
        sum += (x.x + x.y) + (x.z + x.w);
    }
    uint32_t inc = sum;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inc, o);
        if (lane >= o) inc += x;
    }
    if (lane == 31) s_w[warp] = inc;
    __syncthreads();
    // a tile's place in its class: the warp's tiles of the class together
    uint32_t place[8];
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j) {
        const bool in = base + j < ntiles;
        const uint32_t cls = in ? order_class(v[j]) : kOrderClasses;  // past the tiles: a class of its own
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, cls);
        uint32_t at = 0;
        if ((peers & lt) == 0u) at = atomicAdd(&s_cls[cls], (uint32_t)__popc(peers));
        place[j] = __shfl_sync(0xFFFFFFFFu, at, __ffs(peers) - 1) + __popc(peers & lt);
    }
    // low digit: thread (part, d) sums every parts-th of the digit's tiles
    const uint32_t lows = 1u << split.bits[0], parts = 1024u / lows, d = tid & (lows - 1u), part = tid >> split.bits[0];
    uint32_t low = 0;
    for (uint32_t t = part * lows + d; t < ntiles; t += 1024u) low += s_v[t];
    s_low[tid] = low;
    if (warp == 0) {
        uint32_t x = s_w[lane], xi = x;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, xi, o);
            if (lane >= o) xi += y;
        }
        s_w[lane] = xi - x;  // exclusive over warps
    }
    __syncthreads();
    if (warp == 1) {  // first place of each size class, largest class first: lane l takes classes 65 - 3l ..
        uint32_t c[3], s = 0;
#pragma unroll
        for (uint32_t j = 0; j < 3; ++j) {
            const int k = (int)kOrderClasses - 1 - 3 * (int)lane - (int)j;
            c[j] = k >= 0 ? s_cls[k] : 0u;
            s += c[j];
        }
        uint32_t xi = s;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, xi, o);
            if (lane >= o) xi += y;
        }
        uint32_t at = xi - s;
#pragma unroll
        for (uint32_t j = 0; j < 3; ++j) {
            const int k = (int)kOrderClasses - 1 - 3 * (int)lane - (int)j;
            if (k >= 0) s_cls[k] = at;
            at += c[j];
        }
    }
    uint32_t before = 0;  // low digits' exclusive offsets: warps 2 to 9, a digit a thread
    if (warp >= 2 && warp < 10) {
        const uint32_t q = tid - 64u;
        uint32_t x = 0;
        if (q < lows)
            for (uint32_t p = 0; p < parts; ++p) x += s_low[p * lows + q];
        uint32_t xi = x;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, xi, o);
            if (lane >= o) xi += y;
        }
        before = xi - x;
        if (lane == 31) s_lw[warp] = xi;
    }
    __syncthreads();
    if (warp >= 2 && warp < 10 && tid - 64u < lows) {
        for (uint32_t w = 2; w < warp; ++w) before += s_lw[w];
        sort_ctrl->hist[0][tid - 64u] = before;
    }
    uint32_t run = s_w[warp] + inc - sum;
    // the starts take the counts' place (everybody is past reading them), then the order the starts'
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j) {
        const uint32_t t = base + j;
        s_v[t] = run;
        // the first tile of a high digit: the pairs before it
        if (t < ntiles && (t & (lows - 1u)) == 0u) sort_ctrl->hist[1][t >> split.shift[1]] = run;
        place[j] += t < ntiles ? s_cls[order_class(v[j])] : 0u;
        run += v[j];
    }
    if (tid == 1023u) s_v[kScanTilesMax] = run;
    __syncthreads();
    for (uint32_t t = tid; t < ntiles; t += 1024u) ranges[t] = make_uint2(s_v[t], s_v[t + 1]);
    __syncthreads();
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j)
        if (base + j < ntiles) s_v[place[j]] = base + j;
    __syncthreads();
    for (uint32_t t = tid; t < ntiles; t += 1024u) order[t] = s_v[t];
}

// [start, end) of every tile's run in the tile-sorted pairs; each thread checks four
// consecutive pairs with two 16-byte loads.
__global__ void tile_ranges_kernel(const uint2 *pairs, const Ctrl *ctrl, uint2 *ranges,
                                   uint32_t ntiles) {
    frame_kernel_enter();
    const uint32_t n = ctrl->count;
    const uint32_t stride = gridDim.x * blockDim.x * 4u;
    for (uint32_t base = (blockIdx.x * blockDim.x + threadIdx.x) * 4u; base < n; base += stride) {
        uint32_t t[6];  // t[0] = previous pair, t[1..4] = this thread's pairs, t[5] = next pair
        if (base + 4u <= n) {
            const uint4 a = *reinterpret_cast<const uint4 *>(pairs + base);
            const uint4 b = *reinterpret_cast<const uint4 *>(pairs + base + 2);
            t[1] = a.x;
            t[2] = a.z;
            t[3] = b.x;
            t[4] = b.z;
        } else {
            for (uint32_t i = 0; i < 4; ++i) t[1 + i] = base + i < n ? pairs[base + i].x : 0xFFFFFFFFu;
        }
        t[0] = base > 0 ? pairs[base - 1].x : 0xFFFFFFFFu;
        t[5] = base + 4u < n ? pairs[base + 4].x : 0xFFFFFFFFu;
#pragma unroll
        for (uint32_t i = 1; i <= 4; ++i) {
            const uint32_t p = base + i - 1;
            const uint32_t k = t[i];
            if (p >= n || k >= ntiles) continue;
            if (t[i - 1] != k) ranges[k].x = p;
            if (t[i + 1] != k) ranges[k].y = p + 1;
        }
    }
}

// Squared quad offset of the pixel centre (pxc, pyc) from a staged splat, and the alpha there
// (render.wesl:143-181).
__device__ __forceinline__ float fragment_r2(const float4 a, const float4 b, float pxc, float pyc) {
    const float dx = __fsub_rn(pxc, a.x), dy = __fsub_rn(pyc, a.y);
    const float qx = fmaf(b.x, dx, __fmul_rn(b.y, dy));
    const float qy = fmaf(b.z, dx, __fmul_rn(b.w, dy));
    return fmaf(qx, qx, __fmul_rn(qy, qy));
}

template <uint32_t MODE, bool PORTABLE_EXP>
__device__ __forceinline__ float fragment_alpha(const float4 a, float r2, float outline2) {
    if constexpr (MODE == GS_DISPLAY_SPLAT) return __fmul_rn(a.w, PORTABLE_EXP ? exp_portable(-r2) : exp_sfu(-r2));
    return (r2 > outline2) ? 1.0f : a.w;
}

// One fragment of a staged splat at the pixel centre: false when discarded or when it cannot change
// the pixel, else its alpha.
template <uint32_t MODE, bool PORTABLE_EXP>
__device__ __forceinline__ bool fragment(const float4 a, const float4 b, float pxc, float pyc, float outline2,
                                         float *alpha) {
    if constexpr (MODE == GS_DISPLAY_POINT) {
        const float dx = __fsub_rn(pxc, a.x), dy = __fsub_rn(pyc, a.y);
        if (!(dx >= -b.x && dx < b.x && dy >= -b.y && dy < b.y)) return false;
        *alpha = 1.0f;
        return true;
    } else {
        const float r2 = fragment_r2(a, b, pxc, pyc);
        if (!(r2 <= a.z)) return false;
        *alpha = fragment_alpha<MODE, PORTABLE_EXP>(a, r2, outline2);
        return true;
    }
}

// BlendState::ALPHA_BLENDING onto an 8-bit channel, in units of 1/255: round(d·(1-α) + s·α).
__device__ __forceinline__ float blend8(float d, float om, float s_alpha) { return rintf(fmaf(d, om, s_alpha)); }
// The same with two additions for the rounding (exact below 2^22; a blended channel lies in [0, 255]).
constexpr float kRoundBig = 12582912.0f;  // 1.5 * 2^23: a float's last bit there is worth one
__device__ __forceinline__ float blend8_add(float d, float om, float s_alpha) {
    return __fadd_rn(__fadd_rn(fmaf(d, om, s_alpha), kRoundBig), -kRoundBig);
}

// PX: pixels a thread (see raster_tile); a chunk has an entry per thread.
template <uint32_t PX>
struct RasterShared {
    static constexpr uint32_t T = kRasterThreads / PX;
    float4 raw[T * 3];  // the next chunk's splats, thread t's own at 3t
    float4 a[T];        // cx, cy, r² limit, alpha
    float4 b[T];        // q (or the point half sides)
    float4 box[T];      // fragment box in pixel-centre coordinates
    float2 inv[T];      // 1 / |Q·(7, 0)|², 1 / |Q·(0, 4 PX - 1)|² (the block edges in quad space)
    uint32_t kmin;
    uint32_t colours;   // the frame's colour class
};

struct RasterShared1 : RasterShared<1> {
    static constexpr uint32_t PX = 1;
    float4 c[T];  // s255.rgb
    uint8_t list[T / 32][T];
};

// Two pixels a thread: what the blending reads, each value twice for the packed arithmetic; entry T
// is one that no pixel meets.  The lists hold byte offsets into these arrays.
struct RasterShared2 : RasterShared<2> {
    static constexpr uint32_t PX = 2;
    float4 centre[T + 1];   // -cx, -cx, -cy, -cy
    float4 qx[T + 1];       // the first row of q: x, x, y, y
    float4 qy[T + 1];       // the second
    float4 la[T + 1];       // r² limit, alpha, s255.r twice
    float4 gb[T + 1];       // s255.g twice, s255.b twice
    alignas(8) uint32_t list[T / 32][T + 2];
};
template <uint32_t PX>
using RasterSharedOf = typename std::conditional<PX == 1, RasterShared1, RasterShared2>::type;

// The tile's list entries, a chunk at a time, one entry per thread.  The splats of the
// chunk after the staged one are in flight (cp.async into the thread's own part of `raw`) and the
// pair of the chunk after that is in a register, so neither of the two dependent global loads of
// an entry is waited for while the warps blend.
struct ChunkSource {
    const gs_splat *splats;
    const uint32_t *values;  // the tile's own list (RasterJob::values)
    uint32_t value_shift, max_splats;
    uint32_t value;  // pair value of the chunk after the one in flight

    __device__ __forceinline__ uint32_t pair_value(uint32_t base, uint32_t cnt) const {
        return threadIdx.x < cnt ? values[(size_t)(base + threadIdx.x) << value_shift] : 0xFFFFFFFFu;
    }

    template <class Shared>
    __device__ __forceinline__ void fetch(Shared &S, uint32_t k) const {
        float4 *dst = S.raw + 3u * threadIdx.x;
        if (k < max_splats) {  // pair values come from the tile sort; else no entry, or a timeout
            const float4 *src = reinterpret_cast<const float4 *>(splats + k);
            cp_async16(dst, src);
            cp_async16(dst + 1, src + 1);
            cp_async16(dst + 2, src + 2);
        } else {
            dst[0] = make_float4(0.0f, 0.0f, -1.0f, -1.0f);
            dst[1] = dst[2] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }

    // Start a walk: [base, base + cnt) goes into flight, [next, next + next_cnt) is the chunk after.  A walk
    // that ended early left a chunk in flight, whose copies nothing orders with new ones to the same
    // places: they are waited for first.
    template <class Shared>
    __device__ __forceinline__ void begin(Shared &S, uint32_t base, uint32_t cnt, uint32_t next, uint32_t next_cnt) {
        cp_async_wait_all();
        fetch(S, pair_value(base, cnt));
        value = pair_value(next, next_cnt);
    }

    // A splat into the thread's staged entry.
    template <uint32_t MODE, class Shared>
    static __device__ __forceinline__ void put(Shared &S, const float4 a, const float4 b, const float4 c,
                                               float std2) {
        const uint32_t tid = threadIdx.x;
        // Fragments beyond the r² limit cannot change the pixel (see splat_r2_bound).
        const float lim =
            (MODE == GS_DISPLAY_SPLAT) ? splat_r2_bound(c.w, splat_colour_reach(c.x, c.y, c.z), std2) : std2;
        S.a[tid] = make_float4(a.x, a.y, lim, c.w);
        S.b[tid] = b;
        if constexpr (Shared::PX == 1) {
            S.c[tid] = c;
        } else {
            S.centre[tid] = make_float4(-a.x, -a.x, -a.y, -a.y);
            S.qx[tid] = make_float4(b.x, b.x, b.y, b.y);
            S.qy[tid] = make_float4(b.z, b.z, b.w, b.w);
            S.la[tid] = make_float4(lim, c.w, c.x, c.x);
            S.gb[tid] = make_float4(c.y, c.y, c.z, c.z);
        }
        S.box[tid] = make_float4(a.x - a.z, a.x + a.z, a.y - a.w, a.y + a.w);
        if constexpr (MODE != GS_DISPLAY_POINT) {
            const float e1x = b.x * kBlockSpanX, e1y = b.z * kBlockSpanX;
            constexpr float span = 4.0f * Shared::PX - 1.0f;
            const float e2x = b.y * span, e2y = b.w * span;
            S.inv[tid] = make_float2(__frcp_rn(e1x * e1x + e1y * e1y), __frcp_rn(e2x * e2x + e2y * e2y));
        }
    }

    // Stage the chunk in flight (cnt entries), then put the next one (if more) in flight and read the
    // pairs [after, after + after_cnt).  The caller puts a barrier on either side.
    template <uint32_t MODE, class Shared>
    __device__ __forceinline__ void stage(Shared &S, uint32_t cnt, float std2, bool more, uint32_t after,
                                          uint32_t after_cnt) {
        const float4 *raw = S.raw + 3u * threadIdx.x;
        cp_async_wait_all();
        if (threadIdx.x < cnt) put<MODE>(S, raw[0], raw[1], raw[2], std2);
        if (more) {
            fetch(S, value);
            value = pair_value(after, after_cnt);
        }
    }

    // Stage a list that is one chunk, straight from memory.
    template <uint32_t MODE, class Shared>
    __device__ __forceinline__ void stage_only(Shared &S, uint32_t n, float std2) const {
        if (threadIdx.x >= n) return;
        const uint32_t k = pair_value(0, n);
        float4 a = make_float4(0.0f, 0.0f, -1.0f, -1.0f), b = make_float4(0.0f, 0.0f, 0.0f, 0.0f), c = b;
        if (k < max_splats) {
            const float4 *s = reinterpret_cast<const float4 *>(splats + k);
            a = s[0];
            b = s[1];
            c = s[2];
        }
        put<MODE>(S, a, b, c, std2);
    }
};

// Whether the fragment ellipse {p : |Q·(p - c)|² <= lim} of a staged splat meets the rectangle
// of pixel centres [bx0, bx1] x [by0, by1] of a warp's block.  With c outside the
// rectangle, the nearest point of the rectangle in the quadratic norm lies on an edge whose
// half-plane c violates (moving from it toward c must leave the rectangle); Q maps each edge
// to a segment in quad space, where the distance from the origin is minimised in closed form.
// The limit carries a margin (0.2 % + 1e-4) above the rounding of either side, so a block
// holding a pixel centre the fragment test accepts is never dropped; dropping the others
// leaves every pixel unchanged.
__device__ __forceinline__ bool seg_within(float ux, float uy, float ex, float ey, float inv, float lim) {
    float t = -(ux * ex + uy * ey) * inv;
    t = fminf(fmaxf(t, 0.0f), 1.0f);
    const float px = ux + t * ex, py = uy + t * ey;
    return px * px + py * py <= lim;
}

template <uint32_t PX>
__device__ __forceinline__ bool ellipse_meets_block(const float4 a, const float4 q, const float2 inv, float bx0,
                                                    float bx1, float by0, float by1) {
    const bool inx = a.x >= bx0 && a.x <= bx1, iny = a.y >= by0 && a.y <= by1;
    if (inx && iny) return true;
    const float lim = a.z * 1.002f + 1e-4f;
    const float dx = bx0 - a.x, dy = by0 - a.y;
    const float ux = q.x * dx + q.y * dy, uy = q.z * dx + q.w * dy;  // corner (bx0, by0)
    const float e1x = q.x * kBlockSpanX, e1y = q.z * kBlockSpanX;   // along x, 7 px
    constexpr float span = 4.0f * PX - 1.0f;
    const float e2x = q.y * span, e2y = q.w * span;                 // along y, 3 or 7 px
    bool m = false;
    if (!inx) {  // left edge (c left of the block) or right edge
        const bool left = a.x < bx0;
        m = seg_within(left ? ux : ux + e1x, left ? uy : uy + e1y, e2x, e2y, inv.y, lim);
    }
    if (!iny && !m) {  // top edge (c above) or bottom edge
        const bool top = a.y < by0;
        m = seg_within(top ? ux : ux + e2x, top ? uy : uy + e2y, e1x, e1y, inv.x, lim);
    }
    return m;
}

// The calling warp's list of staged entries from jmin on whose fragments can reach its pixel block, in
// draw order: the fragment box, then (splat and ellipse modes) the ellipse itself must meet the block.
template <uint32_t MODE, class Shared>
__device__ __forceinline__ uint32_t compact_chunk(Shared &S, uint32_t jmin, uint32_t cnt, float bx0, float bx1,
                                                  float by0, float by1) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t lt = lanemask_lt();
    uint32_t nl = 0;
    for (uint32_t j0 = jmin & ~31u; j0 < cnt; j0 += 32) {
        const uint32_t j = j0 + lane;
        bool hit = false;
        if (j >= jmin && j < cnt) {
            const float4 box = S.box[j];
            hit = !(box.y < bx0 || box.x > bx1 || box.w < by0 || box.z > by1);
            if (MODE != GS_DISPLAY_POINT && hit)
                hit = ellipse_meets_block<Shared::PX>(S.a[j], S.b[j], S.inv[j], bx0, bx1, by0, by1);
        }
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, hit);
        if constexpr (Shared::PX == 1) {
            if (hit) S.list[warp][nl + __popc(m & lt)] = (uint8_t)j;
        } else {
            if (hit) S.list[warp][nl + __popc(m & lt)] = j * 16u;
        }
        nl += __popc(m);
    }
    if constexpr (Shared::PX == 2) {
        if (lane == 0) S.list[warp][nl] = Shared::T * 16u;  // an even list
    }
    __syncwarp();
    return nl;
}

// A pixel of a warp's block whose transmittance stands for its quarter of the block.
__device__ __forceinline__ float sample_x(uint32_t q) { return (q & 1u) ? 6.0f : 1.0f; }
template <uint32_t PX>
__device__ __forceinline__ float sample_y(uint32_t q) { return PX == 1 ? ((q & 2u) ? 3.0f : 0.0f) : ((q & 2u) ? 6.0f : 1.0f); }

// Two floats in one instruction, each half rounded as the scalar instruction does.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
        "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
        "mul.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
        "add.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
// rintf of both halves: by the conversion unit, or by two packed additions as in blend8_add.
__device__ __forceinline__ float2 rint2_convert(float2 a) { return make_float2(rintf(a.x), rintf(a.y)); }
__device__ __forceinline__ float2 rint2_add(float2 a) {
    return add2(add2(a, make_float2(kRoundBig, kRoundBig)), make_float2(-kRoundBig, -kRoundBig));
}

// Blends the warp's list entries [0, nl) onto the pixel (d), and with BOTH onto the upper bound (h)
// as well, for lanes with `on`.  UNROLL 1: one entry after another, skipping what the fragment test
// skips; the fewest instructions.  UNROLL 4: four entries are evaluated side by side and a missed one
// blends with alpha 0, which leaves the pixel as it is; more instructions, but the warp waits for one
// chain of loads, exp and test where it waited for four, and two channels of three round by additions,
// sooner done than a conversion (2.4M splats at 287x287: 785 -> 760 us a frame, 0.5M in two models at
// 257x192 651 -> 620; all three 767 and 618, but 100k at 640x360 139 -> 141).
template <uint32_t MODE, bool PORTABLE_EXP, bool COUNT, bool BOTH, uint32_t UNROLL>
__device__ __forceinline__ void blend_list(const RasterShared1 &S, uint32_t nl, bool on, float pxc, float pyc,
                                           float outline2, float d[3], float h[3], uint32_t &n_eval, uint32_t &n_alpha,
                                           uint32_t &n_blend) {
    const uint32_t warp = threadIdx.x >> 5;
    auto blend = [&](const float4 c, float al) {
        const float om = __fsub_rn(1.0f, al);
        const float s[3] = {__fmul_rn(c.x, al), __fmul_rn(c.y, al), __fmul_rn(c.z, al)};
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const bool add = UNROLL > 1 && q < 2;  // where the chain of a pixel is waited for
            d[q] = add ? blend8_add(d[q], om, s[q]) : blend8(d[q], om, s[q]);
            if (BOTH) h[q] = add ? blend8_add(h[q], om, s[q]) : blend8(h[q], om, s[q]);
        }
    };
    if constexpr (UNROLL == 1) {
        for (uint32_t i = 0; i < nl; ++i) {
            const uint32_t j = S.list[warp][i];
            float al;
            if (!on) continue;
            if (COUNT) ++n_eval;
            if (!fragment<MODE, PORTABLE_EXP>(S.a[j], S.b[j], pxc, pyc, outline2, &al)) continue;
            if (COUNT) ++n_alpha, n_blend += BOTH ? 2 : 1;
            blend(S.c[j], al);
        }
    } else {
        for (uint32_t i = 0; i < nl; i += UNROLL) {
            float al[UNROLL];
            float4 c[UNROLL];
#pragma unroll
            for (uint32_t u = 0; u < UNROLL; ++u) {
                const uint32_t j = S.list[warp][min(i + u, nl - 1u)];
                const float4 a = S.a[j], b = S.b[j];
                const float r2 = fragment_r2(a, b, pxc, pyc);
                const float v = fragment_alpha<MODE, PORTABLE_EXP>(a, r2, outline2);
                al[u] = (r2 <= a.z && on && i + u < nl) ? v : 0.0f;
                c[u] = S.c[j];
            }
#pragma unroll
            for (uint32_t u = 0; u < UNROLL; ++u) blend(c[u], al[u]);
        }
    }
}

// blend_list for two pixels a thread, (pc.x, pc.y) and (pc.x, pc.z), in packed arithmetic: the list's
// entries two at a time, missed ones blended with alpha 0.  A pixel with a NaN coordinate misses all.
// Bound: the FMA pipe (65 % busy at 1M / 1080p), issue (66 %) and the shared-memory pipe (64 %).
// The rounding is split between the units: all by conversion keeps the conversion unit busy 79 % of
// the time (582 us at 6M / 1080p), all by additions takes 505, two channels of three 489, and two of
// three with both bounds but one of three without 486.  Four entries at a time take 495 us, one 590 (by
// conversion), a test whether any lane hits 589 (by conversion).
template <uint32_t MODE, bool PORTABLE_EXP, bool COUNT, bool BOTH>
__device__ __forceinline__ void blend_list2(const RasterShared2 &S, uint32_t nl, const float3 pc, float outline2,
                                            float2 d[3], float2 h[3], uint32_t &n_eval, uint32_t &n_alpha, uint32_t &n_blend) {
    const uint32_t warp = threadIdx.x >> 5;
    const float2 px = make_float2(pc.x, pc.x), py = make_float2(pc.y, pc.z);
    auto at = [](const float4 *array, uint32_t offset) {
        return *reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(array) + offset);
    };
    auto one = [&](uint32_t offset) {
        const float4 m = at(S.centre, offset), qx = at(S.qx, offset), qy = at(S.qy, offset), la = at(S.la, offset),
                     gb = at(S.gb, offset);
        const float2 dx = add2(px, make_float2(m.x, m.y)), dy = add2(py, make_float2(m.z, m.w));
        const float2 ux = fma2(make_float2(qx.x, qx.y), dx, mul2(make_float2(qx.z, qx.w), dy));
        const float2 uy = fma2(make_float2(qy.x, qy.y), dx, mul2(make_float2(qy.z, qy.w), dy));
        const float2 r2 = fma2(ux, ux, mul2(uy, uy));
        float2 v;
        if constexpr (MODE == GS_DISPLAY_SPLAT && !PORTABLE_EXP) {
            const float2 x = mul2(r2, make_float2(-kLog2E, -kLog2E));
            v.x = __fmul_rn(la.y, exp2_sfu(x.x));
            v.y = __fmul_rn(la.y, exp2_sfu(x.y));
        } else {
            const float4 a = make_float4(0.0f, 0.0f, la.x, la.y);
            v = make_float2(fragment_alpha<MODE, PORTABLE_EXP>(a, r2.x, outline2),
                            fragment_alpha<MODE, PORTABLE_EXP>(a, r2.y, outline2));
        }
        const bool hit0 = r2.x <= la.x, hit1 = r2.y <= la.x;
        if (COUNT) {
            n_eval += (pc.y == pc.y) + (pc.z == pc.z);
            n_alpha += hit0 + hit1, n_blend += (hit0 + hit1) * (BOTH ? 2 : 1);
        }
        const float2 al = make_float2(hit0 ? v.x : 0.0f, hit1 ? v.y : 0.0f);
        const float2 om = fma2(al, make_float2(-1.0f, -1.0f), make_float2(1.0f, 1.0f));
        const float2 s[3] = {mul2(make_float2(la.z, la.w), al), mul2(make_float2(gb.x, gb.y), al),
                             mul2(make_float2(gb.z, gb.w), al)};
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const bool add = q < (BOTH ? 2 : 1);
            d[q] = fma2(d[q], om, s[q]);
            d[q] = add ? rint2_add(d[q]) : rint2_convert(d[q]);
            if (BOTH) {
                h[q] = fma2(h[q], om, s[q]);
                h[q] = add ? rint2_add(h[q]) : rint2_convert(h[q]);
            }
        }
    };
    for (uint32_t i = 0; i < nl; i += 2) {
        const uint2 j = *reinterpret_cast<const uint2 *>(&S.list[warp][i]);
        one(j.x);
        one(j.y);
    }
}

// blend_list2 for frames of kWildColours, whose products with alpha 0 may be NaN and whose blends the
// additions may not round: one entry and pixel at a time, misses passed by.
struct PairState {
    float2 d[3], h[3];
};
template <uint32_t MODE, bool PORTABLE_EXP, bool BOTH>
__device__ __noinline__ PairState blend_list2_wild(const RasterShared2 &S, uint32_t nl, float3 pc, float outline2, PairState P) {
    const uint32_t warp = threadIdx.x >> 5;
    for (uint32_t i = 0; i < nl; ++i) {
        const uint32_t j = S.list[warp][i] / 16u;
        const float4 la = S.la[j], gb = S.gb[j];
        const float c[3] = {la.z, gb.x, gb.z};
        float al;
        if (fragment<MODE, PORTABLE_EXP>(S.a[j], S.b[j], pc.x, pc.y, outline2, &al)) {
            const float om = __fsub_rn(1.0f, al);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const float s = __fmul_rn(c[q], al);
                P.d[q].x = blend8(P.d[q].x, om, s);
                if (BOTH) P.h[q].x = blend8(P.h[q].x, om, s);
            }
        }
        if (fragment<MODE, PORTABLE_EXP>(S.a[j], S.b[j], pc.x, pc.z, outline2, &al)) {
            const float om = __fsub_rn(1.0f, al);
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const float s = __fmul_rn(c[q], al);
                P.d[q].y = blend8(P.d[q].y, om, s);
                if (BOTH) P.h[q].y = blend8(P.h[q].y, om, s);
            }
        }
    }
    return P;
}

// Shortest list that takes the early-out, from the caller's suffix_min (default 1024).  Splats, a pixel
// a thread: three quarters of it (13.5k at 237x133 48 us a frame at 768, 52 at 384).  Two pixels a
// thread walk half as many samples: nine sixteenths (576 by default; compared on one build, 477, 321, 1340
// and 232 us at 6M / 1080p, 1M / 1080p, 3M / 4K and 400k / 1366x768, against 486, 320, 1413, 246 at 768 and
// 480, 330, 1320, 229 at 384).  Ellipses end sooner, as outlines are opaque and interiors keep their full
// alpha: a quarter (256: the frame of 700k at 1600x900 387 us, against 388 at 384, 414 at 768 and 392 at 128).
constexpr float kWalkCourse = 0.9f;
template <uint32_t MODE, uint32_t PX>
__device__ __forceinline__ uint32_t early_out_min(uint32_t suffix_min) {
    if (MODE == GS_DISPLAY_ELLIPSE) return suffix_min / 4u;
    return PX == 2 ? suffix_min / 2u + suffix_min / 16u : suffix_min - suffix_min / 4u;
}

// K4.  One CTA per 16x16 tile; each warp owns an 8x4 pixel block, each thread one pixel, or an 8x8
// block, each thread two pixels of a column (PX; 128 threads a tile, chunks of 128 entries).
// Points are opaque: each pixel takes the nearest point that covers it, found front to back.
// Short tile lists are blended back to front in one pass.  Long ones use an exact early-out:
//   A. walk the list front to back (nearest first) until the transmittance of four sample pixels
//      of the warp's block drops below `eps`, at list position k.  The lanes take 8 splats x 4
//      samples at a time: k only says where to start, so no pixel's own walk is needed;
//   B. blend positions k.. back to front twice, from destination 0 and from 255.  The blend
//      with 8-bit rounding is monotone in the destination, so the two results bound the
//      result of every history before k; when they meet, that is the exact pixel.  (Colours of
//      class k leave histories within +-255 2^k, from which the two start then; wild colours
//      leave none that is bounded, and their lists are blended in one pass.)  A pixel
//      whose bounds do not meet restarts B from k - (n - k) (k = 0 starts from the cleared
//      value, which is exact).
// Every pixel therefore ends bit-identical to the full back-to-front pass.
//
// Bound: the arithmetic of the list loops (no memory system near its limit), so time follows the warp
// iterations and what one of them issues.  Measured at 6M / 1080p, 1M / 1080p and 3M / 4K: 935, 514 and
// 2614 us with a walk A of every pixel over compacted lists and each chunk's loads waited for; 629,
// 392 and 1864 us with the sampled walk, the loads a chunk ahead and exp_sfu; 483, 325 and 1357 us with
// two pixels a thread, which share the list, the loads and, in
// packed instructions, the arithmetic (64 registers, 8 CTAs an SM; 7, 9 and 10 CTAs take 497, 496 and
// 506 us where 8 take 489).  Points (1.5M, 1283x717): 107 us blended like splats, 60 us.
template <uint32_t MODE, bool PORTABLE_EXP, bool COUNT, uint32_t UNROLL, class Shared>
__device__ __forceinline__ void raster_tile(
    Shared &S, const RasterJob &J, const uint32_t *list, uint32_t list_shift, uint32_t n, float std2,
    float outline2, uint32_t suffix_min, float eps, uint32_t colours, unsigned long long *counters, uint32_t tile) {
    // Work tallies of the counting variant (profiling only): fragment evaluations, alphas,
    // channel-triple blends and transmittance updates.
    uint32_t n_eval = 0, n_alpha = 0, n_blend = 0, n_trans = 0;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t W = J.W, H = J.H, tx = tile % J.tiles_x, ty = tile / J.tiles_x;
    constexpr uint32_t PX = Shared::PX;
    const uint32_t wx0 = tx * GS_TILE + (warp & 1u) * 8u, wy0 = ty * GS_TILE + (warp >> 1) * 4u * PX;
    const uint32_t px = wx0 + (lane & 7u), py = wy0 + (lane >> 3);
    const float pxc = (float)px + 0.5f, pyc = (float)py + 0.5f;
    const float bx0 = (float)wx0 + 0.5f, bx1 = (float)wx0 + 7.5f;
    const float by0 = (float)wy0 + 0.5f, by1 = (float)wy0 + 4.0f * PX - 0.5f;
    // the thread's pixels: (px, py) and, with two, (px, py + 4)
    using Value = typename std::conditional<PX == 1, float, float2>::type;
    Value d[3] = {}, h[3] = {};
    const bool wild = colours > kColourClasses;
    const uint32_t early = wild ? 0xFFFFFFFFu : early_out_min<MODE, PX>(suffix_min);
    if (MODE != GS_DISPLAY_POINT && tid == 0) S.colours = colours;  // read after the first barrier
    // blends the list onto the pixels whose `on` is set
    auto blend = [&](auto both, uint32_t nl, const bool *on) {
        if constexpr (PX == 1) {
            if (UNROLL > 1 && wild)
                blend_list<MODE, PORTABLE_EXP, COUNT, decltype(both)::value, 1>(S, nl, on[0], pxc, pyc, outline2, d, h,
                                                                                n_eval, n_alpha, n_blend);
            else
                blend_list<MODE, PORTABLE_EXP, COUNT, decltype(both)::value, UNROLL>(S, nl, on[0], pxc, pyc, outline2, d, h,
                                                                                     n_eval, n_alpha, n_blend);
        } else {
            const float none = __int_as_float(0x7FC00000);
            const float3 pc = make_float3(pxc, on[0] ? pyc : none, on[1] ? pyc + 4.0f : none);
            if (wild) {
                PairState P{{d[0], d[1], d[2]}, {h[0], h[1], h[2]}};
                P = blend_list2_wild<MODE, PORTABLE_EXP, decltype(both)::value>(S, nl, pc, outline2, P);
#pragma unroll
                for (int q = 0; q < 3; ++q) d[q] = P.d[q], h[q] = P.h[q];
                return;
            }
            blend_list2<MODE, PORTABLE_EXP, COUNT, decltype(both)::value>(S, nl, pc, outline2, d, h, n_eval, n_alpha, n_blend);
        }
    };
    if constexpr (PX == 2) {
        if (tid == 0) {  // the entry that fills up a list: read after the first barrier
            S.centre[Shared::T] = S.qx[Shared::T] = S.qy[Shared::T] = S.gb[Shared::T] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            S.la[Shared::T] = make_float4(-1.0f, 0.0f, 0.0f, 0.0f);
        }
    }
    ChunkSource src{J.splats, list, list_shift, J.max_splats, 0u};
    constexpr uint32_t C = Shared::T;
    // the chunk before list position `end` (for walks from the end of the list)
    auto below = [](uint32_t end) { return end > C ? end - C : 0u; };

    if constexpr (MODE == GS_DISPLAY_POINT) {
        // alpha is 1: blending a fragment replaces the pixel, whatever lies behind it
        bool found = px >= W || py >= H;
        auto nearest = [&](uint32_t cnt) {
            const uint32_t nl = compact_chunk<MODE>(S, 0, cnt, bx0, bx1, by0, by1);
            for (int i = (int)nl - 1; i >= 0; --i) {
                const uint32_t j = S.list[warp][i];
                float al;
                if (!found && fragment<MODE, PORTABLE_EXP>(S.a[j], S.b[j], pxc, pyc, outline2, &al)) {
                    const float4 c = S.c[j];
                    d[0] = blend8(0.0f, 0.0f, c.x);
                    d[1] = blend8(0.0f, 0.0f, c.y);
                    d[2] = blend8(0.0f, 0.0f, c.z);
                    found = true;
                }
                if (__all_sync(0xFFFFFFFFu, found)) break;
            }
        };
        if (n <= C) {
            if (n > 0) {
                src.template stage_only<MODE>(S, n, std2);
                __syncthreads();
                nearest(n);
            }
        } else {
            uint32_t base = n - C;
            src.begin(S, base, C, below(base), base - below(base));
            for (uint32_t end = n; end > 0;) {
                src.template stage<MODE>(S, end - base, std2, base > 0, below(below(base)), below(base) - below(below(base)));
                __syncthreads();
                if (__any_sync(0xFFFFFFFFu, !found)) nearest(end - base);
                if (__syncthreads_and(found)) break;
                end = base;
                base = below(end);
            }
            cp_async_wait_all();  // of a walk that ended early
        }
    } else {
        bool all_on[PX];
#pragma unroll
        for (uint32_t p = 0; p < PX; ++p) all_on[p] = true;
        if (n <= C && n < early) {
            if (n > 0) {
                src.template stage_only<MODE>(S, n, std2);
                __syncthreads();
                const uint32_t nl = compact_chunk<MODE>(S, 0, n, bx0, bx1, by0, by1);
                blend(std::false_type(), nl, all_on);
            }
        } else if (n < early) {
            src.begin(S, 0, C, C, min(C, n - C));
            for (uint32_t base = 0; base < n; base += C) {
                const uint32_t cnt = min(C, n - base), after = base + 2u * C;
                src.template stage<MODE>(S, cnt, std2, base + C < n, after, after < n ? min(C, n - after) : 0u);
                __syncthreads();
                const uint32_t nl = compact_chunk<MODE>(S, 0, cnt, bx0, bx1, by0, by1);
                blend(std::false_type(), nl, all_on);
                __syncthreads();
            }
        } else {
            // ---- A: front-to-back transmittance of the samples to find the start position k ----
            uint32_t k = 0;
            {
                const float sxc = bx0 + sample_x(lane & 3u), syc = by0 + sample_y<PX>(lane & 3u);
                float T = 1.0f;  // this lane's share of its sample's transmittance
                bool found = false;
                uint32_t base = below(n), cnt = n - base;
                src.begin(S, base, cnt, below(base), base - below(base));
                for (uint32_t end = n; end > 0;) {
                    src.template stage<MODE>(S, cnt, std2, base > 0, below(below(base)), below(base) - below(below(base)));
                    __syncthreads();
                    for (int top = (int)cnt; top > 0 && !found; top -= 32) {
#pragma unroll
                        for (int it = 0; it < 4; ++it) {
                            const int j = top - 1 - it * 8 - (int)(lane >> 2);
                            float al;
                            if (COUNT && j >= 0) ++n_eval;
                            if (j >= 0 && fragment<MODE, PORTABLE_EXP>(S.a[j], S.b[j], sxc, syc, outline2, &al)) {
                                if (COUNT) ++n_alpha, ++n_trans;
                                // an ellipse's outline is opaque where the sample lies, not where the
                                // block's other pixels do
                                if (MODE == GS_DISPLAY_ELLIPSE) al = S.a[j].w;
                                T = __fmul_rn(T, __fsub_rn(1.0f, al));
                            }
                        }
                        float t = T;  // the product over the sample's eight lanes
                        t *= __shfl_xor_sync(0xFFFFFFFFu, t, 4);
                        t *= __shfl_xor_sync(0xFFFFFFFFu, t, 8);
                        t *= __shfl_xor_sync(0xFFFFFFFFu, t, 16);
                        if (__all_sync(0xFFFFFFFFu, t < eps)) {
                            found = true;
                            k = base + (uint32_t)max(top - 32, 0);
                        }
                    }
                    // A walk that will end in the far part of the list saves nothing: B costs more per
                    // entry than one blend of the whole list.  T falls about evenly per entry, so from a
                    // quarter of the list on it must be on course for eps (to the power kWalkCourse of
                    // the share walked).
                    if (!found && 4u * (n - base) >= n) {
                        float t = T;
                        t *= __shfl_xor_sync(0xFFFFFFFFu, t, 4);
                        t *= __shfl_xor_sync(0xFFFFFFFFu, t, 8);
                        t *= __shfl_xor_sync(0xFFFFFFFFu, t, 16);
                        const float course = __powf(eps, kWalkCourse * (float)(n - base) / (float)n);
                        found = __any_sync(0xFFFFFFFFu, !(t < course));  // k = 0
                    }
                    if (__syncthreads_and(found)) break;
                    end = base;
                    base = below(end);
                    cnt = end - base;
                }
            }
            // ---- B: bounded back-to-front passes from k (the same for all pixels of a warp) ----
            bool active[PX];
#pragma unroll
            for (uint32_t p = 0; p < PX; ++p) active[p] = true;
            auto any_active = [&]() { return active[0] || active[PX - 1]; };
            auto met = [&](uint32_t p) {
                if constexpr (PX == 1) return d[0] == h[0] && d[1] == h[1] && d[2] == h[2];
                else return p == 0 ? d[0].x == h[0].x && d[1].x == h[1].x && d[2].x == h[2].x
                                   : d[0].y == h[0].y && d[1].y == h[1].y && d[2].y == h[2].y;
            };
            for (;;) {
                if (tid == 0) S.kmin = 0xFFFFFFFFu;
                __syncthreads();
                const uint32_t wmin = __reduce_min_sync(0xFFFFFFFFu, any_active() ? k : 0xFFFFFFFFu);
                if (lane == 0 && wmin != 0xFFFFFFFFu) atomicMin(&S.kmin, wmin);
                __syncthreads();
                const uint32_t kmin = S.kmin;
                if (kmin == 0xFFFFFFFFu) break;
                const uint32_t range = S.colours;
                const float top = (k == 0) ? 0.0f : 255.0f * (float)(1u << range), low = range ? -top : 0.0f;
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    if constexpr (PX == 1) {
                        if (active[0]) d[q] = low, h[q] = top;
                    } else {
                        if (active[0]) d[q].x = low, h[q].x = top;
                        if (active[1]) d[q].y = low, h[q].y = top;
                    }
                }
                const uint32_t start = kmin / C * C;
                src.begin(S, start, min(C, n - start), start + C, start + C < n ? min(C, n - start - C) : 0u);
                for (uint32_t base = start; base < n; base += C) {
                    const uint32_t cnt = min(C, n - base), after = base + 2u * C;
                    __syncthreads();
                    src.template stage<MODE>(S, cnt, std2, base + C < n, after, after < n ? min(C, n - after) : 0u);
                    __syncthreads();
                    // wmin is the warp's k: a warp whose suffix starts past this chunk skips it
                    if (wmin < base + C) {
                        const uint32_t nl = compact_chunk<MODE>(S, wmin > base ? wmin - base : 0u, cnt, bx0, bx1, by0, by1);
                        // Bounds that have met stay equal (same inputs, same operations), so once
                        // every started lane of the warp has met, one chain per channel suffices.
                        if (__all_sync(0xFFFFFFFFu, (!active[0] || met(0)) && (!active[PX - 1] || met(PX - 1)))) {
                            blend(std::false_type(), nl, active);
                            // (a pixel that is not active has met before: its bounds are equal as well)
#pragma unroll
                            for (int q = 0; q < 3; ++q) h[q] = d[q];
                        } else {
                            blend(std::true_type(), nl, active);
                        }
                    }
                }
                __syncthreads();
                if (any_active()) {
                    // a pass over the whole list is exact, and the last
                    active[0] = active[0] && k > 0 && !met(0);
                    if (PX == 2) active[PX - 1] = active[PX - 1] && k > 0 && !met(PX - 1);
                    if (any_active()) {
                        const uint32_t suffix = n - k;
                        k = k > suffix ? k - suffix : 0u;
                    }
                }
            }
        }
    }
    auto store = [&](uint32_t y, float r, float g, float b) {
        if (px < W && y < H)
            *reinterpret_cast<uint32_t *>(J.target + (size_t)y * J.pitch + (size_t)px * 4u) =
                (uint32_t)r | ((uint32_t)g << 8) | ((uint32_t)b << 16) | 0xFF000000u;
    };
    if constexpr (PX == 1) {
        store(py, d[0], d[1], d[2]);
    } else {
        store(py, d[0].x, d[1].x, d[2].x);
        store(py + 4u, d[0].y, d[1].y, d[2].y);
    }
    if constexpr (COUNT) {
        const uint32_t v[4] = {n_eval, n_alpha, n_blend, n_trans};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t w = __reduce_add_sync(0xFFFFFFFFu, v[q]);
            if (lane == 0 && w) atomicAdd(counters + q, (unsigned long long)w);
        }
    }
}


// The tile sort keeps its own control block: one thread of a view's rasteriser folds its status into the
// raster's.
__device__ __forceinline__ void merge_status(const RasterJob &J) {
    if (const uint32_t s = J.sort_ctrl->status) atomicOr(&J.ctrl->status, s);
}

// The tile's run of the tile-sorted pairs; empty (and reported) when a scan that gave up left it
// outside the list.
__device__ __forceinline__ uint2 tile_range(const RasterJob &J, uint32_t tile) {
    const uint2 range = J.ranges[tile];
    if (range.y >= range.x && range.y <= J.ctrl->count) return range;
    if (threadIdx.x == 0) atomicOr(&J.ctrl->status, kStatusBounds);
    return make_uint2(0u, 0u);
}

// FEW: a grid of few tiles (at most kFewTiles), whose time is that of its longest lists, not of the
// instructions of all: blend_list four entries at a time, in up to 64 registers a thread (4 CTAs an SM;
// 3 and 5 CTAs take 48 and 55 us for 100k at 640x360, and 4 CTAs 49 us, against 70 us without FEW).
// Pixels a thread: two in packed arithmetic where the instructions count, one for points (a thread
// stops at its first hit) and for grids of few tiles.
template <uint32_t MODE, bool FEW>
constexpr uint32_t kPixels = FEW || MODE == GS_DISPLAY_POINT ? 1u : 2u;
template <uint32_t MODE, bool FEW>
constexpr uint32_t kTileThreads = kRasterThreads / kPixels<MODE, FEW>;
template <uint32_t MODE, bool FEW>
constexpr uint32_t kTileCtas = kPixels<MODE, FEW> == 2 ? 8u : FEW ? 4u : 6u;
template <uint32_t MODE, bool PORTABLE_EXP, bool COUNT, bool FEW>
__global__ void __launch_bounds__(kTileThreads<MODE, FEW>, kTileCtas<MODE, FEW>)
    raster_kernel(const RasterJob J, float std2, float outline2, uint32_t suffix_min, float eps,
                  unsigned long long *counters) {
    __shared__ RasterSharedOf<kPixels<MODE, FEW>> S;
    frame_kernel_enter();
    if (blockIdx.x == 0 && threadIdx.x == 0) merge_status(J);
    const uint32_t tile = J.order ? J.order[blockIdx.x] : blockIdx.x;
    const uint2 r = tile_range(J, tile);
    raster_tile<MODE, PORTABLE_EXP, COUNT, FEW ? 4u : 1u>(S, J, J.values + ((size_t)r.x << J.value_shift), J.value_shift,
                                                          r.y - r.x, std2, outline2, suffix_min, eps, J.ctrl->colours,
                                                          counters, tile);
}

// A direct frame whose pairs do not all fit keeps the first max_pairs of them in draw order, a splat's in
// row-major order of its tiles, as the emission does.  Takes the marks of the ranks past them from
// `hits`; each thread has its own words [first, last).
__device__ __noinline__ void direct_cut(uint32_t *hits, const uint32_t *rects, const uint4 *info, uint32_t ranks,
                                        uint32_t first, uint32_t last, uint32_t tx, uint32_t ty, uint32_t max_pairs,
                                        uint32_t *s_warp) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    auto pairs_of = [&](uint32_t k, const uint4 in) {
        return rects[k] == kEmptyRect ? 0u : in.z ? (uint32_t)__popc(in.z) : (in.y & 0xFFFFu) * (in.y >> 16);
    };
    const uint32_t k0 = 32u * first, k1 = min(ranks, 32u * last);
    uint32_t mine = 0;
    for (uint32_t k = k0; k < k1; ++k) mine += pairs_of(k, info[k]);
    uint32_t incl = mine;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t before = incl - mine;
    for (uint32_t w = 0; w < warp; ++w) before += s_warp[w];
    __syncthreads();
    uint32_t room = max_pairs > before ? max_pairs - before : 0u;
    for (uint32_t k = k0; k < k1; ++k) {
        const uint4 in = info[k];
        const uint32_t c = pairs_of(k, in);
        if (c <= room) {
            room -= c;
            continue;
        }
        const uint32_t dx = tx - (in.x & 0xFFFFu), dy = ty - (in.x >> 16), w = in.y & 0xFFFFu;
        if (dx < w && dy < (in.y >> 16)) {  // else not a tile of it at all
            const uint32_t pos = dy * w + dx, place = in.z ? (uint32_t)__popc(in.z & ((1u << pos) - 1u)) : pos;
            if (place >= room) hits[k / 32u] &= ~(1u << (k & 31u));
        }
        room = 0;
    }
}

// A frame of few splats and tiles without the binning's scan, emission and tile sort: each tile's CTA
// goes through the rectangles of all ranks (draw order), marks those that hold its tile in one bit
// each, and writes its own list of pairs behind those of the CTAs before it.  The scan is bound by L2
// (4 bytes a rank and tile; 16-byte records took 166 us for a frame of 47.5k ranks and 825 tiles, the
// words 102 us), the lists by the latency of a thread's few tile records.
template <uint32_t MODE, bool PORTABLE_EXP, bool FEW>
__global__ void __launch_bounds__(kRasterThreads, FEW ? 4 : 6)
    raster_direct_kernel(const RasterJob J, const uint32_t *rects, const uint4 *info,
                         uint32_t ranks, uint32_t shift, uint32_t *values, uint32_t max_pairs, float std2,
                         float outline2, uint32_t suffix_min, float eps) {
    __shared__ RasterShared1 S;
    __shared__ uint32_t s_warp[kRasterThreads / 32], s_base;
    uint32_t *hits = reinterpret_cast<uint32_t *>(S.raw);  // bit r of word q: rank 32 q + r holds the tile
    static_assert(sizeof(S.raw) * 8 >= kDirectMaxRanks, "a bit per rank");
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, tile = blockIdx.x;
    const uint32_t tx = tile % J.tiles_x, ty = tile / J.tiles_x, words = (ranks + 31u) / 32u;
    const uint32_t here = pack_rect(tx, ty, tx, ty, shift);
    constexpr uint32_t STEP = kRasterThreads / 32u;
    frame_kernel_enter();
    // Both sets' pairs and classes at once, on their way while the ranks are scanned (65k splats at 640x360: 116
    // us a frame through shared memory, 112 so; points, with registers to spare, 98 so and 92 after the scan).
    uint4 sums;
    uint32_t set;
    auto read_sums = [&]() {
        sums = *reinterpret_cast<const uint4 *>(J.ctrl->direct_pairs);
        set = J.ctrl->direct_now;
    };
    if constexpr (MODE != GS_DISPLAY_POINT) read_sums();
    for (uint32_t q0 = warp; q0 < words; q0 += 8u * STEP) {
        uint32_t r[8];
#pragma unroll
        for (uint32_t u = 0; u < 8; ++u) {
            const uint32_t k = 32u * (q0 + u * STEP) + lane;
            r[u] = k < ranks ? rects[k] : kEmptyRect;
        }
#pragma unroll
        for (uint32_t u = 0; u < 8; ++u) {
            const uint32_t q = q0 + u * STEP;
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, rect_may_hold(r[u], here));
            if (lane == 0 && q < words) hits[q] = m;
        }
    }
    if constexpr (MODE == GS_DISPLAY_POINT) read_sums();
    __syncthreads();
    const uint32_t wanted = set ? sums.y : sums.x, colours = set ? sums.w : sums.z;
    if (tile == 0 && tid == 0) {
        J.ctrl->total = wanted;
        if (wanted > max_pairs) atomicOr(&J.ctrl->status, kStatusCapacity);
        J.ctrl->direct_pairs[set ^ 1u] = J.ctrl->direct_class[set ^ 1u] = 0u;
        J.ctrl->direct_next = set ^ 1u;
    }
    // thread t owns the words [t per, (t + 1) per): their places in the list by a block scan
    const uint32_t per = (words + kRasterThreads - 1u) / kRasterThreads;
    const uint32_t first = min(words, tid * per), last = min(words, first + per);
    if (wanted > max_pairs) direct_cut(hits, rects, info, ranks, first, last, tx, ty, max_pairs, s_warp);
    uint32_t sum = 0;
    for (uint32_t q = first; q < last; ++q) {
        const uint32_t found = hits[q];
        uint32_t kept = found;
        for (uint32_t m = found; m; m &= m - 1u) {
            const uint32_t r = __ffs(m) - 1u;
            const uint4 in = info[32u * q + r];  // x0 | y0 << 16, w | h << 16, kept tiles (0: all), value
            const uint32_t dx = tx - (in.x & 0xFFFFu), dy = ty - (in.x >> 16), w = in.y & 0xFFFFu;
            if (!(dx < w && dy < (in.y >> 16)) || (in.z != 0u && !((in.z >> (dy * w + dx)) & 1u))) kept &= ~(1u << r);
        }
        if (kept != found) hits[q] = kept;
        sum += __popc(kept);
    }
    uint32_t incl = sum;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t before = 0, n = 0;
#pragma unroll
    for (uint32_t w = 0; w < kRasterThreads / 32u; ++w) {
        if (w < warp) before += s_warp[w];
        n += s_warp[w];
    }
    if (tid == 0) s_base = n ? atomicAdd(&J.ctrl->count, n) : 0u;
    __syncthreads();
    uint32_t base = s_base;
    if (base > max_pairs || n > max_pairs - base) {  // the lists hold as many pairs as were counted, or fit
        if (tid == 0) atomicOr(&J.ctrl->status, kStatusBounds);
        base = n = 0;
    } else {
        uint32_t at = base + before + incl - sum;
        for (uint32_t q = first; q < last; ++q)
            for (uint32_t m = hits[q]; m; m &= m - 1u) values[at++] = info[32u * q + __ffs(m) - 1u].w;
    }
    __syncthreads();
    raster_tile<MODE, PORTABLE_EXP, false, FEW ? 4u : 1u>(S, J, values + base, 0u, n, std2, outline2, suffix_min, eps, colours,
                                                          nullptr, tile);
}

// One grid over the tiles of several views (a batch): CTA b rasterises tile b - tile_base[v] of
// the view v with tile_base[v] <= b < tile_base[v + 1].
template <uint32_t MODE, bool PORTABLE_EXP>
__global__ void __launch_bounds__(kTileThreads<MODE, false>, kTileCtas<MODE, false>)
    raster_views_kernel(const RasterJob *__restrict__ jobs, const uint32_t *__restrict__ tile_base, uint32_t nviews,
                        float std2, float outline2, uint32_t suffix_min, float eps) {
    __shared__ RasterSharedOf<kPixels<MODE, false>> S;
    frame_kernel_enter();
    uint32_t lo = 0, hi = nviews - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (tile_base[mid] <= blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const RasterJob &J = jobs[lo];
    const uint32_t b = blockIdx.x - tile_base[lo], tile = J.order ? J.order[b] : b;
    if (b == 0 && threadIdx.x == 0) merge_status(J);
    const uint2 r = tile_range(J, tile);
    raster_tile<MODE, PORTABLE_EXP, false, 1u>(S, J, J.values + ((size_t)r.x << J.value_shift), J.value_shift,
                                                          r.y - r.x, std2, outline2, suffix_min, eps, J.ctrl->colours,
                                               nullptr, tile);
}

// Work tallies of the counting raster variant (profiling only).
static __device__ unsigned long long g_raster_counts[4];

cudaError_t raster_counters(unsigned long long out[4], bool reset) {
    cudaError_t e = cudaMemcpyFromSymbol(out, g_raster_counts, sizeof(g_raster_counts));
    if (e == cudaSuccess && reset) {
        const unsigned long long zero[4] = {0, 0, 0, 0};
        e = cudaMemcpyToSymbol(g_raster_counts, zero, sizeof(zero));
    }
    return e;
}

template <uint32_t MODE, bool EXACT, bool COUNT, bool FEW>
static void launch_raster_tiles(const RasterJob &J, float std2, float outline2, cudaStream_t st, const Tuning &t,
                                unsigned long long *counts) {
    launch_frame_kernel(raster_kernel<MODE, EXACT, COUNT, FEW>, J.ntiles, kTileThreads<MODE, FEW>, 0, st,
                        frame_launch_overlaps(st), J, std2, outline2, t.suffix_min, t.eps, counts);
}

// Grids of up to four resident waves of the FEW kernel take it: 1456 tiles (1.4M splats at 892x401)
// 588 -> 544 us a frame, 1881 tiles 271 -> 245 us, 130 tiles with long lists 2453 -> 1997 us; beyond,
// the instructions count: 4836 tiles 169 -> 174 us, 3645 tiles of points 350 -> 356 us.  Views of a
// batch overlap, so the tiles of all of them count.
constexpr uint32_t kFewTiles = 152 * 4 * 4;

template <uint32_t MODE>
static void launch_raster_mode(const RasterJob &J, uint32_t tiles_at_once, float std2, float outline2, int exact,
                               cudaStream_t st, const Tuning &t) {
    const bool few = tiles_at_once <= kFewTiles;
    if (MODE == GS_DISPLAY_SPLAT && !exact && prof_counting()) {
        unsigned long long *counts = nullptr;
        cudaGetSymbolAddress((void **)&counts, g_raster_counts);
        launch_raster_tiles<GS_DISPLAY_SPLAT, false, true, false>(J, std2, outline2, st, t, counts);
    } else if (exact) {
        few ? launch_raster_tiles<MODE, true, false, true>(J, std2, outline2, st, t, nullptr)
            : launch_raster_tiles<MODE, true, false, false>(J, std2, outline2, st, t, nullptr);
    } else {
        few ? launch_raster_tiles<MODE, false, false, true>(J, std2, outline2, st, t, nullptr)
            : launch_raster_tiles<MODE, false, false, false>(J, std2, outline2, st, t, nullptr);
    }
}

template <uint32_t MODE>
static void launch_raster_views_mode(const RasterJob *jobs, const uint32_t *tile_base, uint32_t nviews,
                                     uint32_t total_tiles, float std2, float outline2, int exact, cudaStream_t st,
                                     const Tuning &t) {
    const auto kernel = exact ? raster_views_kernel<MODE, true> : raster_views_kernel<MODE, false>;
    kernel<<<total_tiles, kTileThreads<MODE, false>, 0, st>>>(jobs, tile_base, nviews, std2, outline2, t.suffix_min, t.eps);
}

gs_splat *raster_splat_pool(void *scratch, uint32_t max_splats, uint32_t W, uint32_t H, uint32_t max_pairs) {
    return raster_layout(scratch, max_splats, W, H, max_pairs).splats;
}

RasterJob raster_job(const RasterSegment *segs, uint32_t nseg, uint8_t *target, uint32_t W, uint32_t H,
                     uint32_t pitch, uint32_t max_pairs, void *scratch, bool segmented) {
    uint32_t max_splats = 0;
    for (uint32_t s = 0; s < nseg; ++s) max_splats += segs[s].max_count;
    const RasterLayout L = raster_layout(scratch, max_splats, W, H, max_pairs);
    RasterJob J;
    // Pair values index the model's own splat array (one segment) or the common one.
    J.splats = nseg == 1 ? segs[0].splats : L.splats;
    J.max_splats = nseg == 1 ? segs[0].max_count : max_splats;
    const bool compact = L.value_bits && !segmented;  // else the value is a pair's second word
    J.values = L.items() + (compact ? 0 : 1);
    J.value_shift = compact ? 0u : 1u;
    J.ranges = L.ranges;
    J.order = L.order;
    J.target = target;
    J.W = W;
    J.H = H;
    J.pitch = pitch;
    J.tiles_x = L.tiles_x;
    J.ntiles = L.ntiles;
    J.ctrl = L.ctrl;
    J.sort_ctrl = L.sort_ctrl;
    return J;
}

cudaError_t launch_raster_views(const RasterJob *jobs_dev, const uint32_t *tile_base_dev, uint32_t nviews,
                                uint32_t total_tiles, const RasterMode &u, int exact_exp, cudaStream_t st,
                                const Tuning *tuning) {
    if (nviews == 0 || total_tiles == 0) return cudaSuccess;
    const Tuning tn = tuning ? *tuning : default_tuning();
    const float std2 = u.std_dev * u.std_dev;
    const float o = u.std_dev - 0.1f;
    const float outline2 = o * o;
    prof_mark(kProfRaster, true, st);
    count_launches(1);
    switch (u.display_mode) {
        case GS_DISPLAY_SPLAT:
            launch_raster_views_mode<GS_DISPLAY_SPLAT>(jobs_dev, tile_base_dev, nviews, total_tiles, std2, outline2,
                                                       exact_exp, st, tn);
            break;
        case GS_DISPLAY_ELLIPSE:
            launch_raster_views_mode<GS_DISPLAY_ELLIPSE>(jobs_dev, tile_base_dev, nviews, total_tiles, std2, outline2,
                                                         exact_exp, st, tn);
            break;
        default:
            launch_raster_views_mode<GS_DISPLAY_POINT>(jobs_dev, tile_base_dev, nviews, total_tiles, std2, outline2,
                                                       exact_exp, st, tn);
            break;
    }
    prof_mark(kProfRaster, false, st);
    return cudaGetLastError();
}

cudaError_t launch_binning_front(const RasterSegment *segs, uint32_t nseg, const RasterMode &u, uint32_t W,
                                 uint32_t H, uint32_t max_pairs, void *scratch, cudaStream_t st, bool segmented) {
    uint32_t max_splats = 0;
    for (uint32_t s = 0; s < nseg; ++s) max_splats += segs[s].max_count;
    const RasterLayout L = raster_layout(scratch, max_splats, W, H, max_pairs);
    if (L.ntiles == 0) return cudaSuccess;
    // The first segment with splats clears the arena in its bin_count launch; with none, no kernel
    // reads a flag and the arena mark stays.
    prof_mark(kProfBin, true, st);
    const bool overlap = frame_launch_overlaps(st);
    launch_frame_kernel(raster_init_kernel, 1 + (L.ntiles + 1023) / 1024, 256, 0, st, overlap, L.ctrl,
                        L.sort_ctrl, max_splats ? L.arena_words : kKeepArena, wait_config(), L.counts, L.ntiles);
    count_launches(1);
    const PassSplit split = tile_split(L.key_bits);
    uint32_t rank_offset = 0;
    for (uint32_t s = 0; s < nseg; ++s) {
        const RasterSegment &g = segs[s];
        const uint32_t blocks = (g.max_count + kBinThreads - 1) / kBinThreads;
        if (blocks == 0) continue;
        // a stored tile record is only for the target the preprocess was given
        const uint4 *binfo = g.binfo && g.binfo_w == W && g.binfo_h == H ? g.binfo : nullptr;
        launch_frame_kernel(bin_count_kernel<false>, blocks, kBinThreads, 0, st, overlap, g.splats, binfo, g.sorted_index, g.count,
                            g.max_count, rank_offset, nseg > 1 ? 1 : 0, g.foreign ? 1 : 0, L.tiles_x, L.tiles_y, u.display_mode,
                            u.std_dev * u.std_dev, L.info + rank_offset, L.offsets + rank_offset, L.ctrl,
                            rank_offset ? nullptr : L.flags, nullptr, 0, 0, 0);
        count_launches(1);
        rank_offset += g.max_count;
    }
    // All ranks at once from here on: one segment's live ones, or every segment up to its capacity
    // (ranks without a splat have no tiles).
    const uint32_t *count = nseg == 1 ? segs[0].count : nullptr;
    if (max_splats) {
        launch_frame_kernel(bin_scan_kernel, (max_splats + kScanTile - 1) / kScanTile, 256, 0, st, overlap, L.offsets, count,
                            max_splats, max_pairs, L.ctrl, L.flags);
        count_launches(1);
    }
    // One resident wave at most (and the per-CTA count area): a second, late wave would stretch the
    // kernel; two CTAs an SM at least, as few splats may cover many tiles.
    const size_t emit_smem = L.counting ? (size_t)L.ntiles * 4u : 4u * 256u * 4u;
    const bool compact = L.value_bits && !segmented;
    auto emit = [&](auto kernel) {
        uint32_t wave = resident_ctas(kernel, kBinThreads, emit_smem);
        if (wave == 0 || wave > kEmitBlocks) wave = kEmitBlocks;
        const uint32_t want = std::max((max_splats + kBinThreads - 1) / kBinThreads, 304u), grid = std::min(want, wave);
        launch_frame_kernel(kernel, grid, kBinThreads, emit_smem, st, overlap, L.info, L.offsets, count, max_splats, L.pairs,
                            max_pairs, L.value_bits, L.tiles_x, L.ntiles, L.ctrl, L.sort_ctrl, split, L.blockcounts);
        return grid;
    };
    if (L.counting) {
        const uint32_t grid = compact ? emit(bin_emit_kernel<true, true>) : emit(bin_emit_kernel<true, false>);
        launch_frame_kernel(tile_count_kernel, dim3((L.ntiles + 255) / 256, kCountSlices), 256, 0, st, overlap, L.blockcounts,
                            grid, L.ntiles, L.counts);
        launch_frame_kernel(tile_scan_kernel, 1, 1024, 0, st, overlap, L.counts, L.ntiles, L.ranges, L.order, L.sort_ctrl, split);
        count_launches(3);
    } else {
        compact ? emit(bin_emit_kernel<false, true>) : emit(bin_emit_kernel<false, false>);
        count_launches(1);
    }
    prof_mark(kProfBin, false, st);
    return cudaGetLastError();
}

SortSegment tile_sort_segment(const RasterSegment *segs, uint32_t nseg, uint32_t W, uint32_t H, uint32_t max_pairs,
                              void *scratch) {
    uint32_t max_splats = 0;
    for (uint32_t s = 0; s < nseg; ++s) max_splats += segs[s].max_count;
    const RasterLayout L = raster_layout(scratch, max_splats, W, H, max_pairs);
    const PassSplit split = tile_split(L.key_bits);
    const uint32_t blocks = sort_pairs_blocks(max_pairs);
    SortSegment S;
    S.data = L.pairs;
    S.alt = L.sort_alt;
    S.count = &L.ctrl->count;
    S.max_count = max_pairs;
    for (int p = 0; p < 2; ++p) {
        S.shift[p] = split.shift[p];
        S.bits[p] = split.bits[p];
    }
    S.ctrl = L.sort_ctrl;
    S.owner = L.ctrl;
    S.flags[0] = L.sort_flags;
    S.flags[1] = L.sort_flags + ((size_t)blocks << split.bits[0]);
    return S;
}

bool tile_sort_segmentable(uint32_t W, uint32_t H) {
    const uint32_t tiles = ((W + GS_TILE - 1) / GS_TILE) * ((H + GS_TILE - 1) / GS_TILE);
    return tile_split(bits_for(tiles > 0 ? tiles - 1 : 0)).n == 2;
}

cudaError_t launch_binning_ranges(const RasterSegment *segs, uint32_t nseg, uint32_t W, uint32_t H, uint32_t max_pairs,
                                  void *scratch, cudaStream_t st, bool segmented) {
    uint32_t max_splats = 0;
    for (uint32_t s = 0; s < nseg; ++s) max_splats += segs[s].max_count;
    const RasterLayout L = raster_layout(scratch, max_splats, W, H, max_pairs);
    if (L.ntiles == 0 || L.counting) return cudaSuccess;
    prof_mark(kProfRanges, true, st);
    if (L.value_bits && !segmented) {
        launch_frame_kernel(tile_starts_kernel, 1, 1024, 0, st, frame_launch_overlaps(st), L.counts, L.ntiles, L.ranges);
    } else {
        const cudaError_t e = cudaMemsetAsync(L.ranges, 0, (size_t)L.ntiles * sizeof(uint2), st);
        if (e != cudaSuccess) return e;
        uint32_t rblocks = (max_pairs + 255) / 256;
        if (rblocks > 152 * 8) rblocks = 152 * 8;
        if (rblocks == 0) rblocks = 1;
        launch_frame_kernel(tile_ranges_kernel, rblocks, 256, 0, st, frame_launch_overlaps(st), L.pairs, L.ctrl, L.ranges,
                            L.ntiles);
    }
    prof_mark(kProfRanges, false, st);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_binning(const RasterSegment *segs, uint32_t nseg, const RasterMode &u, uint32_t W, uint32_t H,
                           uint32_t max_pairs, void *scratch, cudaStream_t st) {
    uint32_t max_splats = 0;
    for (uint32_t s = 0; s < nseg; ++s) max_splats += segs[s].max_count;
    const RasterLayout L = raster_layout(scratch, max_splats, W, H, max_pairs);
    if (L.ntiles == 0) return cudaSuccess;
    cudaError_t e = launch_binning_front(segs, nseg, u, W, H, max_pairs, scratch, st);
    if (e != cudaSuccess) return e;
    prof_mark(kProfTileSort, true, st);
    if (L.value_bits)
        e = launch_sort_items(L.items(), L.low(max_pairs), reinterpret_cast<uint32_t *>(L.sort_alt), max_pairs,
                              &L.ctrl->count, L.key_bits, L.value_bits, L.sort_ctrl, L.sort_flags, st,
                              L.counting ? nullptr : L.counts, L.ntiles);
    else
        e = launch_sort_pairs(L.pairs, max_pairs, &L.ctrl->count, L.key_bits, L.sort_ctrl, L.sort_flags, L.sort_alt, st);
    prof_mark(kProfTileSort, false, st);
    if (e != cudaSuccess) return e;
    return launch_binning_ranges(segs, nseg, W, H, max_pairs, scratch, st);
}

// Frames of up to kDirectWork ranks x tiles take raster_direct_kernel: its CTAs read every rank's word,
// where the binning's eight launches and the two of the tile sort cost about 50 us whatever the frame.
// 5k splats x 240 tiles (1.2e6): 95 -> 45 us a frame; 47.5k x 825 (3.9e7): 132 -> 102; 38.9k x 2272
// (8.8e7): 128 -> 125; 68.4k x 1400 (9.6e7): 157 -> 167; 28.6k x 5292 (1.5e8): 135 -> 161.  Views of a
// batch overlap, so the tiles of all of them count (10 views of 11.6k, 4e8 so counted: 234 -> 440).
constexpr uint64_t kDirectWork = 60'000'000;
static bool direct_raster(uint32_t ranks, uint32_t tiles_at_once) {
    return ranks > 0 && ranks <= kDirectMaxRanks && (uint64_t)ranks * tiles_at_once <= kDirectWork;
}

// Frames of separate requests that overlap share the L2 that their scans are bound by: their work
// together is limited too.  Eight served at once, frames/s direct and binned: 12k x 920 tiles (8.8e7
// together) 31,200 and 27,000; 30k x 920 (2.2e8) 24,300 and 24,100; 8k x 3600 (2.3e8) 26,100 and 24,300;
// 16.6k x 3600 (4.8e8) 16,400 and 23,200; 65k x 920 (4.8e8) 13,700 and 20,100.
constexpr uint64_t kDirectWorkInFlight = 240'000'000;

uint64_t direct_raster_work(uint32_t max_splats, uint32_t W, uint32_t H) {
    const uint32_t tiles = ((W + GS_TILE - 1) / GS_TILE) * ((H + GS_TILE - 1) / GS_TILE);
    return direct_raster(max_splats, tiles) ? (uint64_t)max_splats * tiles : 0;
}

template <uint32_t MODE>
static void launch_direct_mode(const RasterJob &J, const RasterLayout &L, uint32_t ranks, uint32_t shift,
                               uint32_t max_pairs, uint32_t tiles_at_once, float std2, float outline2, int exact, cudaStream_t st, const Tuning &t) {
    const bool few = tiles_at_once <= kFewTiles;
    auto go = [&](auto kernel) {
        launch_frame_kernel(kernel, J.ntiles, kRasterThreads, 0, st, frame_launch_overlaps(st), J, L.offsets, L.info, ranks,
                            shift, L.items(), max_pairs, std2, outline2, t.suffix_min, t.eps);
    };
    if (exact) few ? go(raster_direct_kernel<MODE, true, true>) : go(raster_direct_kernel<MODE, true, false>);
    else few ? go(raster_direct_kernel<MODE, false, true>) : go(raster_direct_kernel<MODE, false, false>);
}

// Tile records of every rank, then the tiles (see raster_direct_kernel).
static cudaError_t launch_raster_direct(const RasterSegment *segs, uint32_t nseg, uint32_t ranks, const RasterMode &u,
                                        const RasterJob &J, uint32_t max_pairs, void *scratch, uint32_t tiles_at_once,
                                        int exact_exp, cudaStream_t st, const Tuning &tn) {
    const RasterLayout L = raster_layout(scratch, ranks, J.W, J.H, max_pairs);
    const float std2 = u.std_dev * u.std_dev, o = u.std_dev - 0.1f, outline2 = o * o;
    uint32_t rank_offset = 0, shift = 0;
    while (((L.tiles_x - 1u) >> shift) > 127u || ((L.tiles_y - 1u) >> shift) > 127u) ++shift;
    bool started = false;
    prof_mark(kProfBin, true, st);
    for (uint32_t s = 0; s < nseg; ++s) {
        const RasterSegment &g = segs[s];
        const uint32_t blocks = (g.max_count + kBinThreads - 1) / kBinThreads;
        if (blocks == 0) continue;
        const uint4 *binfo = g.binfo && g.binfo_w == J.W && g.binfo_h == J.H ? g.binfo : nullptr;
        launch_frame_kernel(bin_count_kernel<true>, blocks, kBinThreads, 0, st, frame_launch_overlaps(st), g.splats, binfo,
                            g.sorted_index, g.count, g.max_count, rank_offset, nseg > 1 ? 1 : 0, g.foreign ? 1 : 0, L.tiles_x, L.tiles_y,
                            u.display_mode, std2, L.info + rank_offset, nullptr, L.ctrl, nullptr, L.offsets + rank_offset,
                            shift, started ? 0 : 1, L.arena_words);
        count_launches(1);
        started = true;
        rank_offset += g.max_count;
    }
    prof_mark(kProfBin, false, st);
    prof_mark(kProfRaster, true, st);
    switch (u.display_mode) {
        case GS_DISPLAY_SPLAT:
            launch_direct_mode<GS_DISPLAY_SPLAT>(J, L, ranks, shift, max_pairs, tiles_at_once, std2, outline2, exact_exp, st, tn);
            break;
        case GS_DISPLAY_ELLIPSE:
            launch_direct_mode<GS_DISPLAY_ELLIPSE>(J, L, ranks, shift, max_pairs, tiles_at_once, std2, outline2, exact_exp, st, tn);
            break;
        default:
            launch_direct_mode<GS_DISPLAY_POINT>(J, L, ranks, shift, max_pairs, tiles_at_once, std2, outline2, exact_exp, st, tn);
            break;
    }
    count_launches(1);
    prof_mark(kProfRaster, false, st);
    return cudaGetLastError();
}

cudaError_t launch_raster(const RasterSegment *segs, uint32_t nseg, const RasterMode &u, uint8_t *target,
                          uint32_t W, uint32_t H, uint32_t pitch, uint32_t max_pairs, void *scratch, int exact_exp,
                          cudaStream_t st, const Tuning *tuning, uint32_t tiles_at_once, uint64_t direct_in_flight) {
    const Tuning tn = tuning ? *tuning : default_tuning();
    const RasterJob J = raster_job(segs, nseg, target, W, H, pitch, max_pairs, scratch);
    if (J.ntiles == 0) return cudaSuccess;
    const uint32_t at_once = tiles_at_once > J.ntiles ? tiles_at_once : J.ntiles;
    uint32_t ranks = 0;
    for (uint32_t s = 0; s < nseg; ++s) ranks += segs[s].max_count;
    // (the counting rasteriser and the bounded-wait hook know the general path only)
    if (direct_raster(ranks, at_once) && direct_in_flight <= kDirectWorkInFlight && !prof_counting() && wait_config().stall_tile == kNoStall)
        return launch_raster_direct(segs, nseg, ranks, u, J, max_pairs, scratch, at_once, exact_exp, st, tn);
    cudaError_t e = launch_binning(segs, nseg, u, W, H, max_pairs, scratch, st);
    if (e != cudaSuccess) return e;
    const float std2 = u.std_dev * u.std_dev;
    const float o = u.std_dev - 0.1f;
    const float outline2 = o * o;
    prof_mark(kProfRaster, true, st);
    count_launches(1);
    switch (u.display_mode) {
        case GS_DISPLAY_SPLAT:
            launch_raster_mode<GS_DISPLAY_SPLAT>(J, at_once, std2, outline2, exact_exp, st, tn);
            break;
        case GS_DISPLAY_ELLIPSE:
            launch_raster_mode<GS_DISPLAY_ELLIPSE>(J, at_once, std2, outline2, exact_exp, st, tn);
            break;
        default:
            launch_raster_mode<GS_DISPLAY_POINT>(J, at_once, std2, outline2, exact_exp, st, tn);
            break;
    }
    prof_mark(kProfRaster, false, st);
    return cudaGetLastError();
}

}  // namespace gs
