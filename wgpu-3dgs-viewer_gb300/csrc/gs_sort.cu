// gs_sort.cu — K2: stable LSD onesweep radix sort of u32 keys carrying u32 values.
//
// Same contract as the reference RadixSorter (src/radix_sorter.rs:56-96,658-669; kernels
// src/shader/radix_sort.wgsl:78-529): 8-bit digits, least significant first, stable; the
// reference's 3840-key block stays the unit of the depth buffer's padding.  The GB300 design
// differs: up to 65,536 pairs are sorted by one cluster of CTAs in one launch; larger sorts take pass
// blocks of 2048, 4096 or 7680 keys; one global-histogram kernel reads the keys once
// for all passes (its last CTA turns the histograms into exclusive digit offsets); each pass is
// a single kernel that ranks its block warp by warp (match.any, or one ballot per digit bit, so
// equal digits keep input order), publishes per-digit counts and resolves the block's global
// offsets by decoupled look-back (block = CTA index: CTAs are dispatched in index order, so a
// block waits only for blocks already resident or finished; every wait is bounded all the same),
// then scatters through shared memory so that each digit's run is written contiguously.
// The key count may live in device memory (the preprocess instance count), so a whole frame
// can be enqueued (or graph-captured) without a host round trip.
#include <algorithm>
#include <atomic>
#include <mutex>
#include <utility>

#include "gs300.h"
#include "gs_internal.h"

namespace gs {

// A full pass block is 512 threads x 15 keys = 7680 keys, two of the reference's 3840-key blocks:
// longer digit runs in the scatter, and two CTAs (32 warps) per SM (fewer rows: see sort_rows).  Threads 0..255 own the
// digits in the per-digit phases.  The reordered block (60 KB) lives in dynamic shared memory.
constexpr uint32_t kSortThreads = 512;
constexpr uint32_t kSortRows = 15;
constexpr uint32_t kTileKeys = kSortThreads * kSortRows;  // 7680
constexpr uint32_t kSortWarps = kSortThreads / 32;
constexpr uint32_t kSortCtasPerSm = 2;
constexpr size_t kSortDynSmem = (size_t)kTileKeys * sizeof(uint2);
static_assert(kTileKeys % GS_SORT_BLOCK_KVS == 0, "a pass block covers whole blocks of the reference");

__global__ void ctrl_init_kernel(Ctrl *ctrl, uint32_t arena_words, WaitCfg cfg) {
    frame_kernel_enter();
    ctrl_reset(ctrl, ctrl, arena_words, cfg);
}

__device__ __forceinline__ uint32_t load_count(const uint32_t *count, uint32_t max_count) {
    return count ? min(*count, max_count) : max_count;
}

// Exclusive block scan of one value per thread (WARPS warps).  `tmp` holds WARPS words.
template <uint32_t WARPS>
__device__ __forceinline__ uint32_t block_scan_excl(uint32_t v, uint32_t *tmp, uint32_t *total) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) tmp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t t = lane < WARPS ? tmp[lane] : 0u;
#pragma unroll
        for (uint32_t o = 1; o < WARPS; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, t, o);
            if (lane >= o) t += y;
        }
        if (lane < WARPS) tmp[lane] = t;
    }
    __syncthreads();
    const uint32_t before = warp ? tmp[warp - 1] : 0u;
    *total = tmp[WARPS - 1];
    __syncthreads();
    return before + x - v;
}

// The lanes of the warp whose digit d (below 2^bits, bits <= 8) equals the caller's.  For each digit bit, a
// ballot tells which lanes have it set; those that agree with the caller are ballot ^ flip, flip being
// all ones where the caller's bit is clear, and one three-input operation takes them into the result.  As
// intrinsics the same steps take 98 us for a sort of 2M pairs, 90 so.  Ballots of bits above the digit, zero
// in every lane, change nothing; up to bit 5 they cost less than asking.
__device__ __forceinline__ uint32_t digit_peers(uint32_t d, uint32_t bits) {
    uint32_t peers = 0xFFFFFFFFu;
#pragma unroll
    for (uint32_t b = 0; b < 8; ++b) {
        if (b >= 6 && b >= bits) break;
        asm volatile("{\n\t.reg .pred one;\n\t.reg .b32 bit, flip, voters;\n\t"
                     "and.b32 bit, %1, %2;\n\t"
                     "setp.ne.u32 one, bit, 0;\n\t"
                     "selp.b32 flip, 0, 0xffffffff, one;\n\t"
                     "vote.sync.ballot.b32 voters, one, 0xffffffff;\n\t"
                     "lop3.b32 %0, %0, voters, flip, 0x60;\n\t}"  // a & (b ^ c)
                     : "+r"(peers)
                     : "r"(d), "r"(1u << b));
    }
    return peers;
}

// Global digit histograms of all passes in one read of the keys (four keys per thread and
// iteration, 16-byte loads when the keys are 16-byte aligned).  Low digits are counted with plain
// shared atomics; for the top digit the warp counts the digit of its first lane with one ballot, then
// that of the first lane left, (the high digits of float depth keys take few values, and same-address
// shared atomics would serialise) and the other keys with plain shared atomics.
__device__ __forceinline__ void hist_add(uint32_t *h, uint32_t k, bool valid, const PassSplit &sp, uint32_t hs,
                                         uint32_t lane) {
    // unrolled over the fixed maximum so every field of the split is read at a constant offset
#pragma unroll
    for (uint32_t p = 0; p < kMaxPasses; ++p) {
        if (p >= sp.n) break;
        const uint32_t d = (k >> sp.shift[p]) & ((1u << sp.bits[p]) - 1u);
        if (p + 1 < sp.n) {  // low digits: spread over the bins, rarely equal within a warp
            if (valid) atomicAdd(&h[p * hs + d], 1u);
            continue;
        }
        bool left = valid;
#pragma unroll
        for (uint32_t t = 0; t < 2; ++t) {
            const uint32_t todo = __ballot_sync(0xFFFFFFFFu, left);
            if (!todo) break;
            const uint32_t leader = __ffs(todo) - 1u, dl = __shfl_sync(0xFFFFFFFFu, d, leader);
            const uint32_t same = __ballot_sync(0xFFFFFFFFu, left && d == dl);
            if (lane == leader) atomicAdd(&h[p * hs + dl], (uint32_t)__popc(same));
            left = left && d != dl;
        }
        if (left) atomicAdd(&h[p * hs + d], 1u);
    }
}

// Every CTA first clears its share of the flag-arena words this call must clear (the passes,
// which are the arena's only readers, run after this kernel).
// With `vals`, each CTA also asks L2 for the values of the keys it reads, which the first pass
// reads next (the keys themselves arrive in L2 through this kernel's reads).
// Bound by its chain of steps at middle sizes and by the shared atomics at large ones: 400k, 2M and 6M
// keys 12.2, 17.4 and 31 us with 256 threads a CTA, four waits for keys in a row and the passes' scans one
// after another; 8.5, 13.6 and 28 with four times the threads, the next keys on their way and a warp a scan.
constexpr uint32_t kHistThreads = 1024;
constexpr uint32_t kHistCtas = 152 * 2;  // resident at once
// CTA `block` of the `blocks` that count one sort's keys.
__device__ __forceinline__ void sort_hist_block(const uint32_t *keys, const uint32_t *vals,
                                                const uint32_t *count, uint32_t max_count, const PassSplit &sp,
                                                Ctrl *ctrl, uint64_t *arena, uint32_t block, uint32_t blocks) {
    __shared__ uint32_t h[1024];
    const uint32_t npasses = sp.n, hs = hist_stride(sp.n);
    uint32_t *gh = &ctrl->hist[0][0];
    h[threadIdx.x] = 0u;
    frame_kernel_enter();
    arena_clear(ctrl, arena, block, blocks);
    __syncthreads();
    const uint32_t n = load_count(count, max_count);
    const uint32_t stride = blocks * blockDim.x;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const bool vec = ((uintptr_t)keys & 15u) == 0;
    // Whole warps iterate together (bounds padded to the warp) so the ballots see 32 lanes.
    const uint32_t n4 = (n + 3u) / 4u;
    const uint32_t nr = (n4 + 31u) & ~31u;
    const bool pf = vals && ((uintptr_t)vals & 15u) == 0;
    auto load = [&](uint32_t q, uint32_t k[4]) {
        const uint32_t i0 = q * 4u;
        if (vec && q < nr && i0 + 4u <= n) {
            const uint4 v = *reinterpret_cast<const uint4 *>(keys + i0);
            k[0] = v.x;
            k[1] = v.y;
            k[2] = v.z;
            k[3] = v.w;
        } else {
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) k[j] = q < nr && i0 + j < n ? keys[i0 + j] : 0u;
        }
    };
    uint32_t k[4];
    uint32_t q = block * blockDim.x + threadIdx.x;
    load(q, k);
    for (; q < nr; q += stride) {
        const uint32_t i0 = q * 4u;
        if (pf && threadIdx.x == 0 && i0 < n) {
            // this CTA's 4 x blockDim keys of the iteration start at i0 (a multiple of 16 bytes)
            const uint32_t bytes = min(4u * 4u * blockDim.x, (n - i0) * 4u) & ~15u;
            if (bytes) prefetch_l2_bulk(vals + i0, bytes);
        }
        uint32_t next[4];
        load(q + stride, next);  // under way while this iteration's keys are counted
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) hist_add(h, k[j], i0 + j < n, sp, hs, lane);
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) k[j] = next[j];
    }
    __syncthreads();
    if (const uint32_t v = h[threadIdx.x]) atomicAdd(&gh[threadIdx.x], v);  // the same places in both
    // The last CTA to finish turns the histograms into exclusive digit offsets, once for every
    // block of every pass: a warp a pass.
    __shared__ uint32_t s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&ctrl->ticket[7], 1u) == blocks - 1 ? 1u : 0u;
    __syncthreads();
    if (s_last && warp < npasses) {
        __threadfence();
        const uint32_t digits = 1u << sp.bits[warp];
        uint32_t v[8], sum = 0;
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            v[j] = lane * 8u + j < digits ? __ldcg(&gh[warp * hs + lane * 8u + j]) : 0u;
            sum += v[j];
        }
        uint32_t run = sum;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, run, o);
            if (lane >= o) run += y;
        }
        run -= sum;
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            if (lane * 8u + j < digits) gh[warp * hs + lane * 8u + j] = run;
            run += v[j];
        }
    }
}

__global__ void __launch_bounds__(kHistThreads) sort_hist_kernel(const uint32_t *keys,
                                                                 const uint32_t *vals,
                                                                 const uint32_t *count, uint32_t max_count,
                                                                 const __grid_constant__ PassSplit sp, Ctrl *ctrl,
                                                                 uint64_t *arena) {
    sort_hist_block(keys, vals, count, max_count, sp, ctrl, arena, blockIdx.x, gridDim.x);
}

// Look-back of one digit counter (flags[j * stride], j < tile) that polls up to four
// predecessors per round trip.  The flag word carries everything the reader uses, so relaxed
// loads suffice.  Returns the exclusive prefix; after `limit` polls that find an unpublished
// predecessor it sets the status bit and returns what it has summed.
__device__ __forceinline__ uint32_t look_back_digit(const uint64_t *flags, uint32_t tile, uint32_t epoch,
                                                    uint32_t *status, uint32_t stride, uint32_t limit) {
    uint32_t prefix = 0;
    int64_t j = (int64_t)tile - 1;
    uint32_t spins = 0;
    while (j >= 0) {
        uint64_t w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) w[q] = (j - q >= 0) ? ld_relaxed(flags + (uint64_t)(j - q) * stride) : 0ull;
        bool stalled = false, done = false;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (stalled || done || j < 0) continue;
            const uint32_t st = (uint32_t)(w[q] >> 32) & 3u;
            if ((uint32_t)(w[q] >> 34) != epoch || st == 0u) {
                stalled = true;
                continue;
            }
            prefix += (uint32_t)w[q];
            if (st == kFlagPrefix) done = true;
            else --j;
        }
        if (done) break;
        if (stalled) {
            if (++spins > limit) {
                atomicOr(status, kStatusTimeout);
                break;
            }
            if (spins > 64) __nanosleep(32);
        }
    }
    return prefix;
}

// One LSD pass over the digit at `shift`.  Input and output are either split (keys[],
// values[]) or packed (uint2 {key, value}); packed ping-pong buffers keep each digit's run of
// 8-byte pairs contiguous in the scatter.
// Bound by issue: a row of 32 keys took about 150 instructions of a warp, two thirds of them the
// ballots.  Four a bit (and, setp, vote, not) and no test of the digit width before each, the reorder
// without a check that its own counts make needless, and the output loop five loads deep: 2M random
// pairs 117 -> 103 us, 8M 299 -> 266, tile sort of 24.7M pairs 295 -> 278, depth sort of 6M 213 -> 193.
// MATCH: peers from one match.any instead of a ballot per digit bit.  Measured on GB300 with
// 512-thread blocks, the ballots are the cheaper of the two for both depth keys (0.224 against
// 0.247 ms for a 6M-key sort) and tile keys (0.29 against 0.40 ms).  match.any is a tuning choice
// of the depth sort, and the last pass of float depth keys, whose top digit takes a few values
// per warp, ranks by it.
// The pass of one block (`block`: the look-back tile; lower blocks are lower, earlier-dispatched
// CTAs of the same launch).
template <bool IN_PACKED, bool OUT_PACKED, bool MATCH, uint32_t ROWS = kSortRows>
__device__ __forceinline__ void sort_pass_block(
    const uint32_t *kin, const uint32_t *vin, const uint2 *pin,
    uint32_t *kout, uint32_t *vout, uint2 *pout, const uint32_t *count,
    uint32_t max_count, uint32_t hoff, uint32_t shift, uint32_t digit_bits, Ctrl *ctrl, uint64_t *flags, uint32_t block) {
    constexpr uint32_t KEYS = kSortThreads * ROWS;
    extern __shared__ uint2 s_kv[];  // KEYS pairs (dynamic)
    __shared__ uint32_t s_whist[kSortWarps][256];
    __shared__ uint32_t s_start[256];
    __shared__ uint32_t s_gbase[256];
    __shared__ uint32_t s_tmp[kSortWarps];
    __shared__ uint32_t s_epoch, s_limit, s_stall;

    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, tile = block;
    for (uint32_t k = tid; k < kSortWarps * 256; k += kSortThreads) (&s_whist[0][0])[k] = 0u;
    frame_kernel_enter();
    const uint32_t n = load_count(count, max_count);
    if (tid == 0) {
        s_epoch = *(volatile uint32_t *)&ctrl->epoch;
        s_limit = ctrl->spin_limit;
        s_stall = ctrl->stall_tile;
    }
    // The grid covers the capacity: CTAs past the pairs there are (half of a tile sort's) leave here.
    const uint32_t ntiles = (n + KEYS - 1) / KEYS;
    if (tile >= ntiles) return;
    __syncthreads();
    const uint32_t epoch = s_epoch;
    const uint32_t dmask = (1u << digit_bits) - 1u;  // bits above the key width are ignored
    const uint32_t base = tile * KEYS + warp * (32u * ROWS);

    uint32_t k[ROWS], r[ROWS];
    uint32_t v[IN_PACKED ? ROWS : 1];
#pragma unroll
    for (uint32_t i = 0; i < ROWS; ++i) {
        const uint32_t pos = base + i * 32u + lane;
        const bool ok = pos < n;
        if constexpr (IN_PACKED) {
            const uint2 kv = ok ? pin[pos] : make_uint2(0xFFFFFFFFu, 0u);
            k[i] = kv.x;
            v[i] = kv.y;
        } else {
            k[i] = ok ? kin[pos] : 0xFFFFFFFFu;
        }
    }
    // Warp-local stable ranking: lanes that share a digit form a peer mask (match.any, or one
    // ballot per live digit bit).
    const uint32_t lt = lanemask_lt();
#pragma unroll
    for (uint32_t i = 0; i < ROWS; ++i) {
        const uint32_t d = (k[i] >> shift) & dmask;
        uint32_t peers;
        if constexpr (MATCH) peers = __match_any_sync(0xFFFFFFFFu, d);
        else peers = digit_peers(d, digit_bits);
        const uint32_t rank = __popc(peers & lt);
        const uint32_t pre = s_whist[warp][d];
        __syncwarp();
        if (rank == 0) s_whist[warp][d] = pre + __popc(peers);
        __syncwarp();
        r[i] = pre + rank;
    }
    __syncthreads();

    // Thread d < 256 owns digit d: per-warp exclusive offsets, block count, publication.
    const uint32_t d = tid;
    const bool owner = d < 256u;
    uint32_t run = 0;
    if (owner) {
#pragma unroll
        for (uint32_t w = 0; w < kSortWarps; ++w) {
            const uint32_t c = s_whist[w][d];
            s_whist[w][d] = run;
            run += c;
        }
    }
    const uint32_t total = run;
    const uint32_t invalid = (tile == ntiles - 1) ? ntiles * KEYS - n : 0u;
    // Padding keys (all ones) rank last, in the largest digit.
    const uint32_t pub = (d == dmask) ? total - invalid : total;
    // Digits above dmask hold no key (padding keys sit in digit dmask), so only live digits
    // publish and look back: a pass over 5 live bits keeps 32 flags per block, not 256.
    const bool live = d <= dmask;
    const uint32_t fstride = dmask + 1u;
    uint64_t *f = flags + (size_t)tile * fstride + d;
    if (live) publish_flag(f, tile, s_stall, pack_flag(epoch, tile == 0 ? kFlagPrefix : kFlagAggregate, pub));

    uint32_t blk_total;
    const uint32_t start = block_scan_excl<kSortWarps>(total, s_tmp, &blk_total);
    // the digit's first place in the output: the histograms' producer left exclusive offsets (pass
    // histogram at flat offset hoff; digits above dmask hold no key)
    const uint32_t goff = live ? (&ctrl->hist[0][0])[hoff + d] : 0u;
    uint32_t prefix = 0;
    if (tile > 0 && live) {
        prefix = look_back_digit(flags + d, tile, epoch, &ctrl->status, fstride, s_limit);
        publish_flag(f, tile, s_stall, pack_flag(epoch, kFlagPrefix, prefix + pub));
    }
    if (owner) {
        s_start[d] = start;
        // key j of the reordered block (j >= start for digit d) goes to goff + prefix + (j - start)
        s_gbase[d] = goff + prefix - start;
    }
    __syncthreads();

    // The block's own counts place its KEYS keys (padding included), one to a place.
    if constexpr (IN_PACKED) {
#pragma unroll
        for (uint32_t i = 0; i < ROWS; ++i) {
            const uint32_t dd = (k[i] >> shift) & dmask;
            s_kv[s_start[dd] + s_whist[warp][dd] + r[i]] = make_uint2(k[i], v[i]);
        }
    } else {
        // Values are read only now, after ranking, which keeps them out of registers above.
#pragma unroll
        for (uint32_t i = 0; i < ROWS; ++i) {
            const uint32_t pos = base + i * 32u + lane;
            const uint32_t vv = pos < n ? vin[pos] : 0u;
            const uint32_t dd = (k[i] >> shift) & dmask;
            s_kv[s_start[dd] + s_whist[warp][dd] + r[i]] = make_uint2(k[i], vv);
        }
    }
    __syncthreads();
    const uint32_t valid = min(KEYS, n - tile * KEYS);
    auto put = [&](uint32_t j, const uint2 kv) {
        const uint32_t o = s_gbase[(kv.x >> shift) & dmask] + j;
        if (o < n) {  // always true unless a look-back timed out (status already set)
            if constexpr (OUT_PACKED) {
                pout[o] = kv;
            } else {
                kout[o] = kv.x;
                vout[o] = kv.y;
            }
        }
    };
    if (valid == KEYS) {
#pragma unroll 5
        for (uint32_t i = 0; i < ROWS; ++i) put(tid + i * kSortThreads, s_kv[tid + i * kSortThreads]);
    } else {
        for (uint32_t j = tid; j < valid; j += kSortThreads) put(j, s_kv[j]);
    }
}

// ---- tile sort on compact items ---------------------------------------------------------------
// A pair whose tile id has its low digit taken away fits one word: high digit above the value.  The
// emission writes that word and the low digit as a byte; the first pass sorts words by the bytes, and
// as its output is grouped by the low digit, nobody needs it again; the second sorts by the words' high
// digit and writes the values alone, all that the rasteriser reads of a pair.  5 + 4 + 4 + 4 bytes a
// pair instead of 8 each time, half the registers and shared memory of a pair block (three CTAs an
// SM), and no key to decode twice (6M / 1080p: 278 us as pairs, 228).
// The items are read past L1, as nobody on the SM reads them again (232 -> 229 us).
// TALLY (second pass): also counts each tile's pairs, which the emission does not for targets of many
// tiles.  A block's items have the low digit of the first pass's run they lie in, mostly one for the
// whole block, whose digit counts are then its tiles' counts.
constexpr uint32_t kItemCtasPerSm = 3;
template <bool FIRST>
constexpr size_t kItemDynSmem = kTileKeys * sizeof(uint32_t) + (FIRST ? kTileKeys : 0);

__device__ __forceinline__ uint32_t load_once(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.global.L1::no_allocate.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t load_once(const uint8_t *p) {
    uint32_t v;
    asm volatile("ld.global.L1::no_allocate.u8 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

template <bool FIRST, bool TALLY>
__global__ void __launch_bounds__(kSortThreads, kItemCtasPerSm)
    tile_pass_kernel(const uint32_t *in, const uint8_t *low, uint32_t *out,
                     const uint32_t *count, uint32_t max_count, uint32_t hoff, uint32_t value_bits,
                     uint32_t digit_bits, Ctrl *ctrl, uint64_t *flags, uint32_t low_bits,
                     uint32_t *tile_counts, uint32_t target_tiles) {
    extern __shared__ __align__(16) uint8_t item_smem[];
    uint32_t *s_item = reinterpret_cast<uint32_t *>(item_smem);
    uint8_t *s_low = item_smem + kTileKeys * sizeof(uint32_t);  // FIRST: the digit of each reordered item
    __shared__ uint32_t s_whist[kSortWarps][256];
    __shared__ uint32_t s_start[256];
    __shared__ uint32_t s_gbase[256];
    __shared__ uint32_t s_tmp[kSortWarps];
    __shared__ uint32_t s_epoch, s_limit, s_stall;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, tile = blockIdx.x;
    for (uint32_t k = tid; k < kSortWarps * 256; k += kSortThreads) (&s_whist[0][0])[k] = 0u;
    frame_kernel_enter();
    const uint32_t n = load_count(count, max_count);
    if (tid == 0) {
        s_epoch = *(volatile uint32_t *)&ctrl->epoch;
        s_limit = ctrl->spin_limit;
        s_stall = ctrl->stall_tile;
    }
    const uint32_t ntiles = (n + kTileKeys - 1) / kTileKeys;
    if (tile >= ntiles) return;
    __syncthreads();
    const uint32_t epoch = s_epoch, dmask = (1u << digit_bits) - 1u;
    const uint32_t base = tile * kTileKeys + warp * (32u * kSortRows);

    uint32_t k[kSortRows], r[kSortRows];  // the item; its rank among the warp's of its digit (FIRST: | digit << 16)
#pragma unroll
    for (uint32_t i = 0; i < kSortRows; ++i) {
        const uint32_t pos = base + i * 32u + lane;
        const bool ok = pos < n;  // padding sorts last, in the largest digit
        k[i] = ok ? load_once(in + pos) : 0xFFFFFFFFu;
        if constexpr (FIRST) r[i] = ok ? load_once(low + pos) : dmask;
    }
    const uint32_t lt = lanemask_lt();
#pragma unroll
    for (uint32_t i = 0; i < kSortRows; ++i) {
        const uint32_t d = FIRST ? r[i] : (k[i] >> value_bits) & dmask;
        const uint32_t peers = digit_peers(d, digit_bits);
        const uint32_t rank = __popc(peers & lt);
        const uint32_t pre = s_whist[warp][d];
        __syncwarp();
        if (rank == 0) s_whist[warp][d] = pre + __popc(peers);
        __syncwarp();
        r[i] = pre + rank + (FIRST ? d << 16 : 0u);
    }
    __syncthreads();

    // As sort_pass_block: thread d < 256 owns digit d.
    const uint32_t d = tid;
    const bool owner = d < 256u, live = d <= dmask;
    uint32_t total = 0;
    if (owner) {
#pragma unroll
        for (uint32_t w = 0; w < kSortWarps; ++w) {
            const uint32_t c = s_whist[w][d];
            s_whist[w][d] = total;
            total += c;
        }
    }
    const uint32_t invalid = (tile == ntiles - 1) ? ntiles * kTileKeys - n : 0u;
    const uint32_t pub = (d == dmask) ? total - invalid : total;
    const uint32_t fstride = dmask + 1u;
    uint64_t *f = flags + (size_t)tile * fstride + d;
    if (live) publish_flag(f, tile, s_stall, pack_flag(epoch, tile == 0 ? kFlagPrefix : kFlagAggregate, pub));
    if constexpr (TALLY) {
        __shared__ uint32_t s_run[256];  // first places of the low digits' runs
        const uint32_t lows = 1u << low_bits, at0 = tile * kTileKeys, at1 = min(n, at0 + kTileKeys) - 1u;
        const uint32_t run = tid < lows ? ctrl->hist[0][tid] : 0xFFFFFFFFu;
        if (tid < 256u) s_run[tid] = run;
        // the last run that starts at or before a place holds it
        const uint32_t lo0 = max(1, __syncthreads_count(run <= at0)) - 1u, lo1 = max(1, __syncthreads_count(run <= at1)) - 1u;
        auto tally = [&](uint32_t high, uint32_t lo, uint32_t c) {
            const uint32_t t = (high << low_bits) | lo;
            if (t < target_tiles) atomicAdd(&tile_counts[t], c);
            else atomicOr(&ctrl->status, kStatusBounds);  // pairs of an emission that gave up
        };
        if (lo0 == lo1) {
            if (live && pub) tally(d, lo0, pub);
        } else {
            for (uint32_t i = 0; i < kSortRows; ++i) {
                const uint32_t pos = base + i * 32u + lane;
                if (pos >= n) break;
                uint32_t lo = lo0, hi = lo1;
                while (lo < hi) {
                    const uint32_t mid = (lo + hi + 1u) >> 1;
                    if (s_run[mid] <= pos) lo = mid;
                    else hi = mid - 1u;
                }
                tally((in[pos] >> value_bits) & dmask, lo, 1u);
            }
        }
    }
    uint32_t blk_total;
    const uint32_t start = block_scan_excl<kSortWarps>(total, s_tmp, &blk_total);
    const uint32_t goff = live ? (&ctrl->hist[0][0])[hoff + d] : 0u;  // exclusive digit offsets
    uint32_t prefix = 0;
    if (tile > 0 && live) {
        prefix = look_back_digit(flags + d, tile, epoch, &ctrl->status, fstride, s_limit);
        publish_flag(f, tile, s_stall, pack_flag(epoch, kFlagPrefix, prefix + pub));
    }
    if (owner) {
        s_start[d] = start;
        s_gbase[d] = goff + prefix - start;
    }
    __syncthreads();
    // The block's own counts place its kTileKeys items (padding included), one to a place.
#pragma unroll
    for (uint32_t i = 0; i < kSortRows; ++i) {
        const uint32_t dd = FIRST ? r[i] >> 16 : (k[i] >> value_bits) & dmask;
        const uint32_t at = s_start[dd] + s_whist[warp][dd] + (FIRST ? r[i] & 0xFFFFu : r[i]);
        s_item[at] = k[i];
        if constexpr (FIRST) s_low[at] = (uint8_t)dd;
    }
    __syncthreads();
    const uint32_t valid = min(kTileKeys, n - tile * kTileKeys), vmask = (1u << value_bits) - 1u;
    auto put = [&](uint32_t j) {
        const uint32_t item = s_item[j];
        const uint32_t dd = FIRST ? s_low[j] : (item >> value_bits) & dmask;
        const uint32_t o = s_gbase[dd] + j;
        if (o < n) out[o] = FIRST ? item : item & vmask;  // false only where a look-back timed out (status set)
    };
    if (valid == kTileKeys) {
#pragma unroll 5
        for (uint32_t i = 0; i < kSortRows; ++i) put(tid + i * kSortThreads);
    } else {
        for (uint32_t j = tid; j < valid; j += kSortThreads) put(j);
    }
}

template <bool IN_PACKED, bool OUT_PACKED, bool MATCH, uint32_t ROWS = kSortRows>
__global__ void __launch_bounds__(kSortThreads, kSortCtasPerSm) sort_pass_kernel(
    const uint32_t *kin, const uint32_t *vin, const uint2 *pin,
    uint32_t *kout, uint32_t *vout, uint2 *pout, const uint32_t *count,
    uint32_t max_count, uint32_t hoff, uint32_t shift, uint32_t digit_bits, Ctrl *ctrl, uint64_t *flags) {
    // look-back predecessors are lower, earlier-dispatched CTAs
    sort_pass_block<IN_PACKED, OUT_PACKED, MATCH, ROWS>(kin, vin, pin, kout, vout, pout, count, max_count, hoff, shift,
                                                  digit_bits, ctrl, flags, blockIdx.x);
}

// One pass of many independent packed pair sorts in a single launch (a segmented sort): segment v
// owns the CTAs [block_base[v], block_base[v + 1]) and each of them runs the pass on a block of
// that segment's pairs with the segment's own control block, digit offsets and look-back flags.
// Pass 0 reads `data` and writes `alt`, pass 1 the reverse, so two passes leave the pairs in place.
__global__ void __launch_bounds__(kSortThreads, kSortCtasPerSm)
    sort_segments_kernel(const SortSegment *__restrict__ segs, const uint32_t *__restrict__ block_base, uint32_t nseg,
                         uint32_t pass) {
    uint32_t lo = 0, hi = nseg - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (block_base[mid] <= blockIdx.x) lo = mid;
        else hi = mid - 1;
    }
    const SortSegment &S = segs[lo];
    const uint2 *in = pass ? S.alt : S.data;
    uint2 *out = pass ? S.data : S.alt;
    sort_pass_block<true, true, false>(nullptr, nullptr, in, nullptr, nullptr, out, S.count, S.max_count,
                                       pass * hist_stride(2), S.shift[pass], S.bits[pass], S.ctrl, S.flags[pass], blockIdx.x - block_base[lo]);
}

// Several independent depth sorts, each launch over all of them: sort v owns the CTAs [block0[v],
// block0[v + 1]) of a pass and hist0[v].. of the histogram.  One sort after another leaves the chip
// idle at the end of every launch (6M keys in four models: 325 us, 181 together).
constexpr uint32_t kSortGroup = 8;
struct SortGroup {
    PassSplit sp;
    uint32_t n;
    uint32_t hist0[kSortGroup + 1], block0[kSortGroup + 1];
    DepthSort sort[kSortGroup];
    Ctrl *ctrl[kSortGroup];
    uint64_t *flags[kSortGroup];
    uint32_t flag_words[kSortGroup];
    uint2 *a[kSortGroup], *b[kSortGroup];  // packed buffers
};

__device__ __forceinline__ uint32_t group_member(const uint32_t *first, uint32_t n) {
    uint32_t v = 0;
    while (v + 1 < n && first[v + 1] <= blockIdx.x) ++v;
    return v;
}

__global__ void ctrl_init_group_kernel(const __grid_constant__ SortGroup G, WaitCfg cfg) {
    frame_kernel_enter();
    ctrl_reset(G.ctrl[blockIdx.x], G.ctrl[blockIdx.x], G.flag_words[blockIdx.x], cfg);
}

__global__ void __launch_bounds__(kHistThreads) sort_hist_group_kernel(const __grid_constant__ SortGroup G) {
    const uint32_t v = group_member(G.hist0, G.n);
    const DepthSort &s = G.sort[v];
    sort_hist_block(s.keys, s.vals, s.count, s.max_count, G.sp, G.ctrl[v], G.flags[v], blockIdx.x - G.hist0[v],
                    G.hist0[v + 1] - G.hist0[v]);
}

// Pass p: the first reads the split keys and values and writes a, the others go from a to b and back, the
// last writes the split arrays.
template <bool IN_PACKED, bool OUT_PACKED, bool MATCH>
__global__ void __launch_bounds__(kSortThreads, kSortCtasPerSm)
    sort_pass_group_kernel(const __grid_constant__ SortGroup G, uint32_t p) {
    const uint32_t v = group_member(G.block0, G.n);
    const DepthSort &s = G.sort[v];
    uint64_t *flags = G.flags[v];
    for (uint32_t q = 0; q < p; ++q) flags += (size_t)(G.block0[v + 1] - G.block0[v]) << G.sp.bits[q];
    uint2 *from = (p & 1u) ? G.a[v] : G.b[v], *to = (p & 1u) ? G.b[v] : G.a[v];
    sort_pass_block<IN_PACKED, OUT_PACKED, MATCH>(s.keys, s.vals, from, s.keys, s.vals, to, s.count, s.max_count,
                                                  p * hist_stride(G.sp.n), G.sp.shift[p], G.sp.bits[p], G.ctrl[v], flags,
                                                  blockIdx.x - G.block0[v]);
}

// Each segment's sort status into the control block of the area it belongs to.
__global__ void merge_segments_status_kernel(const SortSegment *segs, uint32_t nseg) {
    for (uint32_t v = threadIdx.x; v < nseg; v += blockDim.x) atomicOr(&segs[v].owner->status, segs[v].ctrl->status);
}

__global__ void unpack_pairs_kernel(const uint2 *src, uint32_t *kd, uint32_t *vd, const uint32_t *count,
                                    uint32_t max_count) {
    frame_kernel_enter();
    const uint32_t n = load_count(count, max_count);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint2 kv = src[i];
        kd[i] = kv.x;
        vd[i] = kv.y;
    }
}

__global__ void copy_packed_kernel(const uint2 *src, uint2 *dst, const uint32_t *count, uint32_t max_count) {
    frame_kernel_enter();
    const uint32_t n = load_count(count, max_count);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[i] = src[i];
}

static inline uint32_t sort_passes(uint32_t key_bits) { return (key_bits + 7u) / 8u; }
// Live bits of pass p's digit: keys are below 2^key_bits.  Invalid (padding) keys are all ones
// but sort last either way, because they hold the largest value in every live bit.
PassSplit even_split(uint32_t key_bits) {
    PassSplit sp{};
    sp.n = sort_passes(key_bits);
    const uint32_t base = sp.n ? key_bits / sp.n : 0u, extra = sp.n ? key_bits % sp.n : 0u;
    uint32_t at = 0;
    for (uint32_t p = 0; p < sp.n; ++p) {
        sp.shift[p] = at;
        sp.bits[p] = base + (p < extra ? 1u : 0u);
        at += sp.bits[p];
    }
    return sp;
}

// Passes of a tile-pair sort: two passes up to 16 key bits (a target of up to 65536 tiles), so the
// pairs of every such view end where they started and views can share one segmented launch.
PassSplit tile_split(uint32_t key_bits) {
    if (key_bits > 16) return even_split(key_bits);
    PassSplit sp{};
    sp.n = 2;
    sp.bits[0] = (key_bits + 1) / 2;
    sp.bits[1] = key_bits / 2;
    sp.shift[0] = 0;
    sp.shift[1] = sp.bits[0];
    return sp;
}

// Passes of `key_bits` in digits of at most max_digit bits, spread evenly.
PassSplit even_split_max(uint32_t key_bits, uint32_t max_digit) {
    PassSplit sp{};
    sp.n = (key_bits + max_digit - 1) / max_digit;
    if (sp.n > kMaxPasses) sp.n = kMaxPasses;
    const uint32_t base = sp.n ? key_bits / sp.n : 0u, extra = sp.n ? key_bits % sp.n : 0u;
    uint32_t at = 0;
    for (uint32_t p = 0; p < sp.n; ++p) {
        sp.shift[p] = at;
        sp.bits[p] = base + (p < extra ? 1u : 0u);
        at += sp.bits[p];
    }
    return sp;
}

// Digit widths the split-array sort can be run with (Tuning::sort_digit_bits).
constexpr uint32_t kMinDigitBits = 6, kMaxDigitBits = 8;

static size_t sort_tiles(uint32_t max_count, uint32_t rows = kSortRows) {
    const size_t keys = (size_t)kSortThreads * rows, t = (max_count + keys - 1) / keys;
    return t ? t : 1;
}

// Look-back flags of a sort: per pass, one word per block and live digit ([tiles][2^bits]).
static size_t sort_flag_words(uint32_t max_count, const PassSplit &sp, uint32_t rows = kSortRows) {
    size_t w = 0;
    for (uint32_t p = 0; p < sp.n; ++p) w += sort_tiles(max_count, rows) << sp.bits[p];
    return w;
}

struct SortLayout {
    Ctrl *ctrl;
    uint64_t *flags;  // the area's flag arena
    uint2 *alt_a, *alt_b;
    uint32_t ntiles;
    size_t flag_words;
};

// Scratch: control block | flag arena (look-back flags of every pass) | packed buffer A | packed
// buffer B (split sorts of 3+ passes only).  The control block and the arena start at offsets no
// call size moves; the buffers after the arena follow its size.  A sort in small blocks has no buffer B: its
// longer arena (768 or 1024 words for 2048 keys) ends in that buffer's 8 bytes a key.
static SortLayout sort_layout(void *scratch, uint32_t max_count, const PassSplit &sp, uint32_t rows = kSortRows) {
    SortLayout L;
    uint8_t *p = reinterpret_cast<uint8_t *>(scratch);
    L.ntiles = (uint32_t)sort_tiles(max_count, rows);
    L.ctrl = reinterpret_cast<Ctrl *>(p);
    p += align_up(sizeof(Ctrl), 256);
    L.flags = reinterpret_cast<uint64_t *>(p);
    L.flag_words = sort_flag_words(max_count, sp, rows);
    p += align_up(L.flag_words * sizeof(uint64_t), 256);
    L.alt_a = reinterpret_cast<uint2 *>(p);
    p += align_up((size_t)max_count * 8, 256);
    L.alt_b = reinterpret_cast<uint2 *>(p);
    return L;
}

// Sized for the widest layout over every digit width a call may use, so a caller's scratch fits
// whatever width the tuning picks.
size_t sort_scratch_bytes(uint32_t max_count, uint32_t key_bits) {
    size_t flags = 0;
    uint32_t np = 0;
    for (uint32_t db = kMinDigitBits; db <= kMaxDigitBits; ++db) {
        const PassSplit sp = even_split_max(key_bits, db);
        const size_t f = sort_flag_words(max_count, sp);
        if (f > flags) flags = f;
        if (sp.n > np) np = sp.n;
    }
    return align_up(sizeof(Ctrl), 256) + align_up(flags * sizeof(uint64_t), 256) +
           (np >= 3 ? 2 : 1) * align_up((size_t)max_count * 8, 256);
}

static uint32_t grid_for(uint32_t max_count) {
    uint32_t blocks = (max_count + 255) / 256;
    if (blocks > 152 * 8) blocks = 152 * 8;
    return blocks ? blocks : 1;
}

// MATCH_LAST: the last pass ranks by match.any whatever MATCH says (the top digit of float depth
// keys takes a few values per warp, where one match.any is cheaper than a ballot per bit).
template <bool MATCH, bool MATCH_LAST>
static void launch_sort_passes(uint32_t *keys, uint32_t *vals, uint32_t max_count, const uint32_t *count,
                               const PassSplit &sp, const SortLayout &L, cudaStream_t st) {
    const uint32_t npasses = sp.n, hs = hist_stride(sp.n);
    const bool overlap = frame_launch_overlaps(st);
    uint64_t *f = L.flags;
    if (npasses == 1) {
        launch_frame_kernel(sort_pass_kernel<false, true, MATCH>, L.ntiles, kSortThreads, kSortDynSmem, st, overlap, 
            keys, vals, nullptr, nullptr, nullptr, L.alt_a, count, max_count, 0, sp.shift[0], sp.bits[0], L.ctrl, f);
        launch_frame_kernel(unpack_pairs_kernel, grid_for(max_count), 256, 0, st, overlap, L.alt_a, keys, vals, count, max_count);
        count_launches(2);
        return;
    }
    uint2 *src = L.alt_a, *dst = L.alt_b;
    launch_frame_kernel(sort_pass_kernel<false, true, MATCH>, L.ntiles, kSortThreads, kSortDynSmem, st, overlap, 
        keys, vals, nullptr, nullptr, nullptr, src, count, max_count, 0, sp.shift[0], sp.bits[0], L.ctrl, f);
    f += (size_t)L.ntiles << sp.bits[0];
    for (uint32_t p = 1; p + 1 < npasses; ++p) {
        launch_frame_kernel(sort_pass_kernel<true, true, MATCH>, L.ntiles, kSortThreads, kSortDynSmem, st, overlap, 
            nullptr, nullptr, src, nullptr, nullptr, dst, count, max_count, p * hs, sp.shift[p], sp.bits[p], L.ctrl, f);
        f += (size_t)L.ntiles << sp.bits[p];
        uint2 *t = src;
        src = dst;
        dst = t;
    }
    launch_frame_kernel(sort_pass_kernel<true, false, MATCH || MATCH_LAST>, L.ntiles, kSortThreads, kSortDynSmem, st, overlap, 
        nullptr, nullptr, src, keys, vals, nullptr, count, max_count, (npasses - 1) * hs, sp.shift[npasses - 1],
        sp.bits[npasses - 1], L.ctrl, f);
    count_launches(npasses);
}

// Passes of a small sort, an even number: from the split arrays to A and back, ROWS rows a block.
template <bool MATCH_LAST, uint32_t ROWS>
static void launch_small_passes(uint32_t *keys, uint32_t *vals, uint32_t max_count, const uint32_t *count,
                                const PassSplit &sp, const SortLayout &L, cudaStream_t st) {
    const uint32_t hs = hist_stride(sp.n);
    const size_t smem = (size_t)kSortThreads * ROWS * sizeof(uint2);
    const bool overlap = frame_launch_overlaps(st);
    uint64_t *f = L.flags;
    for (uint32_t p = 0; p < sp.n; ++p) {
        auto go = [&](auto kernel) {
            launch_frame_kernel(kernel, L.ntiles, kSortThreads, smem, st, overlap, keys, vals, L.alt_a, keys, vals, L.alt_a,
                                count, max_count, p * hs, sp.shift[p], sp.bits[p], L.ctrl, f);
        };
        if (p % 2 == 0) go(sort_pass_kernel<false, true, false, ROWS>);
        else if (p + 1 < sp.n) go(sort_pass_kernel<true, false, false, ROWS>);
        else go(sort_pass_kernel<true, false, MATCH_LAST, ROWS>);
        f += (size_t)L.ntiles << sp.bits[p];
    }
    count_launches(sp.n);
}

// The pass kernels take kSortDynSmem of dynamic shared memory, above the default 48 KB a launch
// may ask for: allow it once per device, before the first launch there.
static cudaError_t ensure_sort_smem() {
    static std::atomic<uint64_t> ready{0};  // bit d: device d's pass kernels allow kSortDynSmem
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const uint64_t bit = dev < 64 ? (1ull << dev) : 0ull;
    if (bit && (ready.load(std::memory_order_acquire) & bit)) return cudaSuccess;
    const void *fns[] = {
        (const void *)sort_pass_kernel<false, true, false>, (const void *)sort_pass_kernel<true, true, false>,
        (const void *)sort_pass_kernel<true, false, false>, (const void *)sort_pass_kernel<false, true, true>,
        (const void *)sort_pass_kernel<true, true, true>,   (const void *)sort_pass_kernel<true, false, true>,
        (const void *)sort_segments_kernel,
        (const void *)sort_pass_kernel<false, true, false, 8>, (const void *)sort_pass_kernel<true, false, false, 8>,
        (const void *)sort_pass_kernel<true, false, true, 8>,
        (const void *)sort_pass_group_kernel<false, true, false>, (const void *)sort_pass_group_kernel<true, true, false>,
        (const void *)sort_pass_group_kernel<true, false, true>,
    };
    for (const void *f : fns) {
        e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSortDynSmem);
        if (e != cudaSuccess) return e;
    }
    const std::pair<const void *, size_t> items[] = {
        {(const void *)tile_pass_kernel<true, false>, kItemDynSmem<true>},
        {(const void *)tile_pass_kernel<false, false>, kItemDynSmem<false>},
        {(const void *)tile_pass_kernel<false, true>, kItemDynSmem<false>},
    };
    for (const auto &f : items) {
        e = cudaFuncSetAttribute(f.first, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)f.second);
        if (e != cudaSuccess) return e;
    }
    ready.fetch_or(bit, std::memory_order_acq_rel);
    return cudaSuccess;
}

// ---- small sorts: every pass in one launch of one cluster --------------------------------------
// Up to 65,536 pairs (16 CTAs of 4 rows) are sorted by a single thread-block cluster: CTA c holds positions
// [c K, (c + 1) K) in registers (K = 1024 ROWS), each pass ranks them as sort_pass_block does, the
// CTAs exchange their digit counts through distributed shared memory, and every pair goes straight
// to its place in the shared memory of the CTA that owns it.  Two cluster barriers a pass take the
// place of a launch, a look-back and a trip through global memory, and the digit histogram kernel
// falls away, as a pass counts what it holds.
constexpr uint32_t kClusterThreads = 1024;
constexpr uint32_t kClusterWarps = kClusterThreads / 32;
constexpr uint32_t kClusterMaxCtas = 16;
constexpr uint32_t kClusterMaxPairs = kClusterMaxCtas * kClusterThreads * 4;

template <uint32_t ROWS>
struct ClusterShared {
    uint2 kv[kClusterThreads * ROWS];
    uint32_t whist[kClusterWarps][256];
    uint32_t cnt[kClusterMaxCtas][256];
    uint32_t part[4][256];
    uint32_t base[256];
    uint32_t tmp[kClusterWarps];
};

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
// Every CTA of the cluster arrives; shared-memory writes before it, local and remote, are visible
// after it.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The shared address `p` of this CTA, in CTA `cta` of the cluster.
__device__ __forceinline__ uint32_t remote_smem(const void *p, uint32_t cta) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(cta));
    return r;
}

template <uint32_t ROWS>
__global__ void __launch_bounds__(kClusterThreads, 1)
    sort_cluster_kernel(uint32_t *keys, uint32_t *vals, const uint32_t *count,
                        uint32_t max_count, const PassSplit sp, Ctrl *ctrl) {
    constexpr uint32_t K = kClusterThreads * ROWS;
    extern __shared__ __align__(16) uint8_t cluster_smem[];
    ClusterShared<ROWS> &S = *reinterpret_cast<ClusterShared<ROWS> *>(cluster_smem);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, lt = lanemask_lt();
    const uint32_t me = cluster_rank(), ctas = cluster_size();
    frame_kernel_enter();
    if (me == 0 && tid == 0) ctrl->status = 0u;  // of the call; no flag is waited for here
    const uint32_t n = load_count(count, max_count);
    const bool some = me * K < n;  // this CTA holds pairs
    const uint32_t at0 = warp * (32u * ROWS) + lane;

    uint32_t k[ROWS], v[ROWS], r[ROWS];
#pragma unroll
    for (uint32_t i = 0; i < ROWS; ++i) {
        const uint32_t pos = me * K + at0 + 32u * i;
        const bool ok = pos < n;  // padding keys (all ones, last) stay behind every pair
        k[i] = ok ? keys[pos] : 0xFFFFFFFFu;
        v[i] = ok ? vals[pos] : 0u;
    }
    cluster_sync();  // every CTA has started: its shared memory may be written
    for (uint32_t p = 0; p < sp.n; ++p) {
        const uint32_t shift = sp.shift[p], bits = sp.bits[p], dmask = (1u << bits) - 1u;
        for (uint32_t q = tid; q < kClusterWarps * 256u; q += kClusterThreads) (&S.whist[0][0])[q] = 0u;
        __syncthreads();
        if (some) {
#pragma unroll
            for (uint32_t i = 0; i < ROWS; ++i) {
                const uint32_t d = (k[i] >> shift) & dmask;
                const uint32_t peers = digit_peers(d, bits);
                const uint32_t rank = __popc(peers & lt);
                const uint32_t pre = S.whist[warp][d];
                __syncwarp();
                if (rank == 0) S.whist[warp][d] = pre + __popc(peers);
                __syncwarp();
                r[i] = pre + rank;
            }
        }
        __syncthreads();
        // Digit d of warps 8q .. 8q + 7 (q = tid / 256): exclusive offsets over the warps, the CTA's count
        const uint32_t d = tid & 255u, q = tid >> 8;
        uint32_t c[8], sum = 0;
#pragma unroll
        for (uint32_t w = 0; w < 8; ++w) {
            c[w] = S.whist[8u * q + w][d];
            sum += c[w];
        }
        S.part[q][d] = sum;
        __syncthreads();
        uint32_t run = 0, total = 0;
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            const uint32_t x = S.part[j][d];
            if (j < q) run += x;
            total += x;
        }
#pragma unroll
        for (uint32_t w = 0; w < 8; ++w) {
            S.whist[8u * q + w][d] = run;
            run += c[w];
        }
        for (uint32_t j = q; j < ctas; j += 4)
            asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote_smem(&S.cnt[me][d], j)), "r"(total) : "memory");
        cluster_sync();  // also: every CTA holds its pairs in registers, so kv is free
        uint32_t all = 0, before = 0;
        if (tid < 256u) {
            for (uint32_t j = 0; j < ctas; ++j) {
                const uint32_t x = S.cnt[j][d];
                if (j < me) before += x;
                all += x;
            }
        }
        uint32_t every;
        const uint32_t first = block_scan_excl<kClusterWarps>(all, S.tmp, &every);
        if (tid < 256u) S.base[d] = first + before;
        __syncthreads();
        if (some) {
#pragma unroll
            for (uint32_t i = 0; i < ROWS; ++i) {
                const uint32_t dd = (k[i] >> shift) & dmask;
                const uint32_t pos = S.base[dd] + S.whist[warp][dd] + r[i];  // below the pairs of all CTAs
                const uint32_t cta = pos / K;
                asm volatile("st.shared::cluster.v2.u32 [%0], {%1, %2};" ::"r"(remote_smem(&S.kv[pos - cta * K], cta)),
                             "r"(k[i]), "r"(v[i])
                             : "memory");
            }
        }
        cluster_sync();
        if (some) {
#pragma unroll
            for (uint32_t i = 0; i < ROWS; ++i) {
                const uint2 kv = S.kv[at0 + 32u * i];
                k[i] = kv.x;
                v[i] = kv.y;
            }
        }
    }
#pragma unroll
    for (uint32_t i = 0; i < ROWS; ++i) {
        const uint32_t pos = me * K + at0 + 32u * i;
        if (pos < n) {
            keys[pos] = k[i];
            vals[pos] = v[i];
        }
    }
}

// Largest cluster of sort_cluster_kernel<ROWS> that the current device can hold (0: none).
template <uint32_t ROWS>
static uint32_t cluster_ctas_supported() {
    constexpr int kDevices = 64;
    static std::atomic<int> cached[kDevices];  // 1 + the answer
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) return 0;
    int known = cached[dev].load(std::memory_order_acquire);
    if (known) return (uint32_t)(known - 1);
    auto *fn = sort_cluster_kernel<ROWS>;
    uint32_t best = 0;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ClusterShared<ROWS>)) == cudaSuccess &&
        cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
        for (uint32_t ctas = kClusterMaxCtas; ctas >= 1 && !best; ctas /= 2) {
            cudaLaunchAttribute attr{};
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x = ctas;
            attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(ctas);
            cfg.blockDim = dim3(kClusterThreads);
            cfg.dynamicSmemBytes = sizeof(ClusterShared<ROWS>);
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) == cudaSuccess && clusters > 0) best = ctas;
        }
    }
    cudaGetLastError();  // an unsupported size is not the caller's error
    cached[dev].store((int)best + 1, std::memory_order_release);
    return best;
}

// Whether a sort goes to one cluster, where the tuning's sort knobs have nothing to choose.
template <uint32_t ROWS>
static bool cluster_holds(uint32_t max_count) {
    return max_count > 0 && (max_count - 1) / (kClusterThreads * ROWS) < cluster_ctas_supported<ROWS>();
}
bool sort_in_cluster(uint32_t max_count) {
    return cluster_holds<1>(max_count) || cluster_holds<2>(max_count) || cluster_holds<4>(max_count);
}

// Launches the sort on one cluster where `max_count` fits ROWS rows; false: not this size.
template <uint32_t ROWS>
static bool launch_cluster_rows(uint32_t *keys, uint32_t *vals, uint32_t max_count, const uint32_t *count,
                                const PassSplit &sp, Ctrl *ctrl, cudaStream_t st, cudaError_t *err) {
    constexpr uint32_t K = kClusterThreads * ROWS;
    if (!cluster_holds<ROWS>(max_count)) return false;
    const uint32_t ctas = (max_count + K - 1) / K;
    cudaLaunchAttribute attr[2] = {};
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = sizeof(ClusterShared<ROWS>);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = frame_launch_overlaps(st) ? 2 : 1;
    *err = cudaLaunchKernelEx(&cfg, sort_cluster_kernel<ROWS>, keys, vals, count, max_count, sp, ctrl);
    count_launches(1);
    return true;
}

// The fewest rows that fit: fewer rows a thread and more CTAs are faster throughout (16384 pairs: 24.5,
// 25.0 and 29.2 us at 1, 2 and 4 rows).  Against the histogram and pass kernels, with the launches of
// either overlapped: 40,000 pairs 29.0 us, 39.9; 65,536 pairs 32.4, 43.4; with 8 rows 70,000 pairs would
// take 45.1, 43.0 and 131,072 pairs 51.2, 45.4.
static bool launch_sort_cluster(uint32_t *keys, uint32_t *vals, uint32_t max_count, const uint32_t *count,
                                uint32_t key_bits, Ctrl *ctrl, cudaStream_t st, cudaError_t *err) {
    const PassSplit sp = even_split(key_bits);
    return launch_cluster_rows<1>(keys, vals, max_count, count, sp, ctrl, st, err) ||
           launch_cluster_rows<2>(keys, vals, max_count, count, sp, ctrl, st, err) ||
           launch_cluster_rows<4>(keys, vals, max_count, count, sp, ctrl, st, err);
}

static PassSplit pass_split(uint32_t key_bits, const Tuning &tn) {
    return even_split_max(key_bits, std::max(kMinDigitBits, std::min(kMaxDigitBits, tn.sort_digit_bits)));
}

// Four keys a thread, up to one resident wave.
static uint32_t hist_grid(uint32_t max_count, const Tuning &tn) {
    if (tn.hist_blocks) return std::min(tn.hist_blocks, 152u * 8u);
    return std::min((max_count + kHistThreads * 4 - 1) / (kHistThreads * 4), kHistCtas);
}

// Rows of a pass block.  A block of 15 rows keeps one SM's issue slots busy for about 4.5 us, so sorts that
// leave SMs without a block take fewer rows: up to 96 blocks of 4 (70,000 pairs 42.5 -> 31.3 us, 131,072
// 44.5 -> 34.4, 200,000 46.5 -> 38.8, 38.4 with 8 rows), up to 400 blocks of 8 (400,000 50.4 -> 44.9, 1M
// 75.7 -> 64.5, 1.4M 86.2 -> 77.0; 2M 91.4 -> 100).  2 rows are slower throughout, 6 in between.  Sorts that
// run at the same time (a batch's views) fill the SMs together, so the keys of all of them count.
// Never more scratch than sort_scratch_bytes asks for: sorts of 9 to 12 key bits have one packed buffer
// there, which leaves a longer arena no room.
constexpr uint32_t kRows4Keys = 96 * 4 * kSortThreads, kRows8Keys = 400 * 8 * kSortThreads;
static uint32_t sort_rows(uint32_t max_count, uint64_t keys_at_once, uint32_t key_bits, const PassSplit &sp, const Tuning &tn) {
    // an even number of passes, which ends in the split arrays without a second packed buffer
    if (sp.n % 2 != 0 || tn.sort_match) return kSortRows;
    const uint32_t rows = keys_at_once <= kRows4Keys ? 4u : keys_at_once <= kRows8Keys ? 8u : kSortRows;
    const size_t bytes = align_up(sizeof(Ctrl), 256) + align_up(sort_flag_words(max_count, sp, rows) * sizeof(uint64_t), 256) +
                         align_up((size_t)max_count * 8, 256);
    return bytes <= sort_scratch_bytes(max_count, key_bits) ? rows : kSortRows;
}

cudaError_t launch_sort(uint32_t *keys, uint32_t *vals, uint32_t max_count, const uint32_t *count,
                        uint32_t key_bits, void *scratch, cudaStream_t st, int prof_stage, const Tuning *tuning,
                        uint64_t keys_at_once) {
    // One cluster where the pairs fit (the bounded-wait hook stalls look-backs, which it has none of).
    if (wait_config().stall_tile == kNoStall) {
        cudaError_t e = cudaSuccess;
        prof_mark(prof_stage, true, st);
        const bool done = launch_sort_cluster(keys, vals, max_count, count, key_bits, reinterpret_cast<Ctrl *>(scratch), st, &e);
        if (done) prof_mark(prof_stage, false, st);
        if (done) return e == cudaSuccess ? cudaGetLastError() : e;
    }
    if (cudaError_t e = ensure_sort_smem(); e != cudaSuccess) return e;
    const Tuning tn = tuning ? *tuning : default_tuning();
    const PassSplit sp = pass_split(key_bits, tn);
    const uint32_t rows = sort_rows(max_count, std::max<uint64_t>(keys_at_once, max_count), key_bits, sp, tn);
    const SortLayout L = sort_layout(scratch, max_count, sp, rows);
    const bool overlap = frame_launch_overlaps(st);
    // With no pairs no kernel reads the flags, and none clears them: the arena mark stays.
    launch_frame_kernel(ctrl_init_kernel, 1, 256, 0, st, overlap, L.ctrl, max_count ? (uint32_t)L.flag_words : kKeepArena,
                                        wait_config());
    count_launches(1);
    if (max_count == 0) return cudaGetLastError();
    prof_mark(prof_stage, true, st);
    const uint32_t hist_blocks = hist_grid(max_count, tn);
    launch_frame_kernel(sort_hist_kernel, hist_blocks, kHistThreads, 0, st, overlap, keys, vals, count, max_count, sp, L.ctrl, L.flags);
    count_launches(1);
    // Keys of kDepthKeyBits are the render path's float depth keys (1 - ndc.z).
    if (rows == 4)
        key_bits == kDepthKeyBits ? launch_small_passes<true, 4>(keys, vals, max_count, count, sp, L, st)
                                  : launch_small_passes<false, 4>(keys, vals, max_count, count, sp, L, st);
    else if (rows == 8)
        key_bits == kDepthKeyBits ? launch_small_passes<true, 8>(keys, vals, max_count, count, sp, L, st)
                                  : launch_small_passes<false, 8>(keys, vals, max_count, count, sp, L, st);
    else if (tn.sort_match)
        launch_sort_passes<true, true>(keys, vals, max_count, count, sp, L, st);
    else if (key_bits == kDepthKeyBits)
        launch_sort_passes<false, true>(keys, vals, max_count, count, sp, L, st);
    else
        launch_sort_passes<false, false>(keys, vals, max_count, count, sp, L, st);
    prof_mark(prof_stage, false, st);
    return cudaGetLastError();
}

static cudaError_t launch_sort_group(const SortGroup &G, cudaStream_t st) {
    if (cudaError_t e = ensure_sort_smem(); e != cudaSuccess) return e;
    const bool overlap = frame_launch_overlaps(st);
    const uint32_t blocks = G.block0[G.n];
    launch_frame_kernel(ctrl_init_group_kernel, G.n, 256, 0, st, overlap, G, wait_config());
    prof_mark(kProfDepthSort, true, st);
    launch_frame_kernel(sort_hist_group_kernel, G.hist0[G.n], kHistThreads, 0, st, overlap, G);
    launch_frame_kernel(sort_pass_group_kernel<false, true, false>, blocks, kSortThreads, kSortDynSmem, st, overlap, G, 0u);
    for (uint32_t p = 1; p + 1 < G.sp.n; ++p)
        launch_frame_kernel(sort_pass_group_kernel<true, true, false>, blocks, kSortThreads, kSortDynSmem, st, overlap, G, p);
    launch_frame_kernel(sort_pass_group_kernel<true, false, true>, blocks, kSortThreads, kSortDynSmem, st, overlap, G,
                        G.sp.n - 1);
    prof_mark(kProfDepthSort, false, st);
    count_launches(2 + G.sp.n);
    return cudaGetLastError();
}

// Sorts of more pairs than a cluster holds go together, up to kSortGroup at a time (with sort_match, which
// the grouped passes have no variant for, one by one).
cudaError_t launch_depth_sorts(const DepthSort *sorts, uint32_t n, cudaStream_t st) {
    SortGroup G{};
    const Tuning tn = default_tuning();
    G.sp = pass_split(kDepthKeyBits, tn);
    uint32_t only = 0;  // the sort that the group began with
    auto flush = [&]() {
        cudaError_t e = cudaSuccess;
        if (G.n == 1) {
            const DepthSort &s = sorts[only];
            e = launch_sort(s.keys, s.vals, s.max_count, s.count, kDepthKeyBits, s.scratch, st);
        } else if (G.n > 1) {
            e = launch_sort_group(G, st);
        }
        G.n = 0;
        return e;
    };
    for (uint32_t i = 0; i < n; ++i) {
        const DepthSort &s = sorts[i];
        cudaError_t e = cudaSuccess;
        if (s.max_count <= kClusterMaxPairs || tn.sort_match) {
            e = launch_sort(s.keys, s.vals, s.max_count, s.count, kDepthKeyBits, s.scratch, st);
        } else {
            const SortLayout L = sort_layout(s.scratch, s.max_count, G.sp);
            const uint32_t v = G.n++;
            if (v == 0) only = i;
            G.sort[v] = s;
            G.ctrl[v] = L.ctrl;
            G.flags[v] = L.flags;
            G.flag_words[v] = (uint32_t)L.flag_words;
            G.a[v] = L.alt_a;
            G.b[v] = L.alt_b;
            G.hist0[v + 1] = G.hist0[v] + hist_grid(s.max_count, tn);
            G.block0[v + 1] = G.block0[v] + L.ntiles;
            if (G.n == kSortGroup) e = flush();
        }
        if (e != cudaSuccess) return e;
    }
    return flush();
}

size_t sort_pairs_flag_words(uint32_t max_count, uint32_t key_bits) {
    return sort_flag_words(max_count, tile_split(key_bits));
}

uint32_t sort_pairs_blocks(uint32_t max_count) { return (uint32_t)sort_tiles(max_count); }

cudaError_t launch_sort_segments(const SortSegment *segs_dev, const uint32_t *block_base_dev, uint32_t nseg,
                                 uint32_t total_blocks, cudaStream_t st) {
    if (nseg == 0 || total_blocks == 0) return cudaSuccess;
    if (cudaError_t e = ensure_sort_smem(); e != cudaSuccess) return e;
    for (uint32_t pass = 0; pass < 2; ++pass)
        sort_segments_kernel<<<total_blocks, kSortThreads, kSortDynSmem, st>>>(segs_dev, block_base_dev, nseg, pass);
    merge_segments_status_kernel<<<1, 256, 0, st>>>(segs_dev, nseg);
    count_launches(3);
    return cudaGetLastError();
}

cudaError_t launch_sort_pairs(uint2 *data, uint32_t max_count, const uint32_t *count, uint32_t key_bits, Ctrl *ctrl,
                              uint64_t *flags, uint2 *alt, cudaStream_t st) {
    const PassSplit split = tile_split(key_bits);
    if (max_count == 0) return cudaSuccess;
    if (cudaError_t e = ensure_sort_smem(); e != cudaSuccess) return e;
    const uint32_t ntiles = (uint32_t)sort_tiles(max_count);
    const bool overlap = frame_launch_overlaps(st);
    uint2 *src = data, *dst = alt;
    uint64_t *f = flags;
    for (uint32_t p = 0; p < split.n; ++p) {
        launch_frame_kernel(sort_pass_kernel<true, true, false>, ntiles, kSortThreads, kSortDynSmem, st, overlap, nullptr, nullptr, src, nullptr, nullptr, dst,
                                                                            count, max_count, p * hist_stride(split.n),
                                                                            split.shift[p],
                                                                            split.bits[p], ctrl, f);
        f += (size_t)ntiles << split.bits[p];
        uint2 *t = src;
        src = dst;
        dst = t;
    }
    count_launches(split.n);
    if (split.n & 1u) {
        launch_frame_kernel(copy_packed_kernel, grid_for(max_count), 256, 0, st, overlap, src, data, count, max_count);
        count_launches(1);
    }
    return cudaGetLastError();
}

cudaError_t launch_sort_items(uint32_t *items, const uint8_t *low, uint32_t *alt, uint32_t max_count, const uint32_t *count,
                              uint32_t key_bits, uint32_t value_bits, Ctrl *ctrl, uint64_t *flags, cudaStream_t st,
                              uint32_t *tile_counts, uint32_t target_tiles) {
    const PassSplit split = tile_split(key_bits);
    if (max_count == 0) return cudaSuccess;
    if (cudaError_t e = ensure_sort_smem(); e != cudaSuccess) return e;
    const uint32_t ntiles = (uint32_t)sort_tiles(max_count);
    const bool overlap = frame_launch_overlaps(st);
    uint64_t *flags1 = flags + ((size_t)ntiles << split.bits[0]);
    launch_frame_kernel(tile_pass_kernel<true, false>, ntiles, kSortThreads, kItemDynSmem<true>, st, overlap, items, low, alt,
                        count, max_count, 0, value_bits, split.bits[0], ctrl, flags, 0, nullptr, 0);
    launch_frame_kernel(tile_counts ? tile_pass_kernel<false, true> : tile_pass_kernel<false, false>, ntiles, kSortThreads,
                        kItemDynSmem<false>, st, overlap, alt, nullptr, items, count, max_count, hist_stride(2), value_bits,
                        split.bits[1], ctrl, flags1, split.bits[0], tile_counts, target_tiles);
    count_launches(2);
    return cudaGetLastError();
}

// ---- allocation-free sort entry point -------------------------------------------------------
// Scratch for gs_radix_sort_no_alloc lives in this file-scope device array instead of memory the
// caller provides, so that entry point never allocates.  It holds the largest layout the entry
// point accepts (kNoAllocMaxPairs pairs of 32-bit keys, four passes) and every device that loads
// the library holds it until the process exits.  A __device__ array without an initialiser is
// zero when the module loads, which is the state a fresh scratch area needs; after that, calls of
// any size and key width reuse it as any caller scratch is reused (the flag arena sits at a fixed
// offset and is cleared where a call's layout grows past the previous one).
constexpr uint32_t kNoAllocMaxPairs = 1u << 20;
constexpr size_t kNoAllocTiles = (kNoAllocMaxPairs + kTileKeys - 1) / kTileKeys;
constexpr size_t kNoAllocBytes = ((sizeof(Ctrl) + 255) / 256) * 256 +
                                 ((4 * kNoAllocTiles * 256 * sizeof(uint64_t) + 255) / 256) * 256 +
                                 2 * (((size_t)kNoAllocMaxPairs * 8 + 255) / 256) * 256;
static __device__ __align__(256) unsigned char g_no_alloc_scratch[kNoAllocBytes];

namespace {
std::mutex g_no_alloc_mu;
constexpr int kNoAllocDevices = 64;
void *g_no_alloc_ptr[kNoAllocDevices] = {};
}  // namespace

// Device address of the array on the current device.  In host code the array's name is only a
// stand-in, not a device address: the first call on a device looks the address up with that
// device current and caches it; later calls reuse it.
static cudaError_t no_alloc_scratch(void **out) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kNoAllocDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> g(g_no_alloc_mu);
    if (!g_no_alloc_ptr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_no_alloc_scratch);
        if (e != cudaSuccess) return e;
        g_no_alloc_ptr[dev] = p;
    }
    *out = g_no_alloc_ptr[dev];
    return cudaSuccess;
}

}  // namespace gs

extern "C" gs_status gs_radix_sort_no_alloc(uint32_t *keys, uint32_t *values, uint32_t max_count,
                                            const uint32_t *count, uint32_t key_bits, gs_stream stream) {
    using namespace gs;
    if (key_bits < 1 || key_bits > 32) return set_error(GS_ERR_INVALID_ARG, "gs_radix_sort_no_alloc: key_bits not in 1..=32");
    if (max_count > kNoAllocMaxPairs)
        return set_error(GS_ERR_INVALID_ARG,
                         "gs_radix_sort_no_alloc: max_count exceeds the static scratch limit of 1048576 pairs "
                         "(use gs_radix_sort with caller scratch)");
    if (max_count && (!keys || !values)) return set_error(GS_ERR_INVALID_ARG, "gs_radix_sort_no_alloc: NULL buffer");
    if (sort_scratch_bytes(max_count, key_bits) > kNoAllocBytes)
        return set_error(GS_ERR_INVALID_ARG, "gs_radix_sort_no_alloc: layout exceeds the static scratch");
    cudaStream_t st = (cudaStream_t)stream;
    void *scratch = nullptr;
    cudaError_t e = no_alloc_scratch(&scratch);
    if (e == cudaSuccess) e = launch_sort(keys, values, max_count, count, key_bits, scratch, st);
    if (e != cudaSuccess) return set_error(GS_ERR_CUDA, cudaGetErrorString(e));
    return GS_OK;
}
