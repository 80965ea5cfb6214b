// The tile sort: the (tile, depth, index) order of all splat-tile pairs made per tile, for frames of
// at least kTileSortEntries entries that do not crowd on few tiles (Plan::by_tile). Where the LSD chain (sort.cu) sorts the visible entries by depth
// over the whole frame and then distributes them, here the pairs are distributed first and each
// tile's list is sorted by itself, in shared memory:
//   1. the preprocess cuts each visible entry's rectangle to the tiles its pixel bounds reach and counts
//      them (one add per pair, no result waited for);
//   2. tile_scan turns the counts into the tiles' ranges;
//   3. tile_scatter appends every pair (depth key, entry) to its tile's list, in any order;
//   4. tile_sort sorts each list by (depth key, entry) -- no two pairs of a tile are equal, so the order
//      is unique and does not depend on the order of arrival: it is the reference's order. Lists of
//      more than kTileChunk pairs are sorted in chunks, and tile_merge merges each chunk with the other
//      chunks of its list for its pairs' places.
// Four short kernels (five for scenes of more Gaussians than a group of chunks holds, one more for
// more tiles than one scan CTA adds up) where the chain has thirteen to eighteen, each latency-bound at a
// few microseconds, and every pair is written twice instead of three to five times. Measured, frame
// time with the chain -> with the tile sort: 87 -> 53 us (100k Gaussians, 640x360), 253 -> 217 us (740k,
// 1280x720), 536 -> 483 us (2.2M, 1920x1080), the 64-view 1M batch 7.35 -> 7.04 ms; with the rectangles
// cut 47, 197, 447 us and 6.42 ms.
//
// No CTA waits on another. What bounds the parts: the scatter its scattered accesses (an add and an
// 8-byte store per pair, each a sector of its own: 46 pairs a nanosecond over the chip), the sort and
// the scan latency. The counters lie kTileStride words
// apart: neighbouring tiles are hit together (the 100k view takes 72, 59, 55, 53 us at 1, 2, 4, 8 words;
// several counters per tile, to spread the adds further, cost the scan more than they gave).
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace ab2 {
namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

// ---- ranges ------------------------------------------------------------------------------------

constexpr int kScanThreads = 1024;
constexpr int kScanPer = 4;
constexpr unsigned kScanTiles = kScanThreads * kScanPer;  // tiles per scan CTA
// Up to this many tiles a scan CTA adds up the counts before its own itself; above it, tile_sums_kernel
// leaves each CTA's total first.
constexpr unsigned kScanDirect = 1u << 16;

// sums[b] = pairs of tiles [b kScanTiles, (b + 1) kScanTiles).
__global__ void __launch_bounds__(kScanThreads) tile_sums_kernel(const unsigned* __restrict__ counts, unsigned tiles,
                                                                 unsigned* __restrict__ sums) {
    chain_entry();
    __shared__ unsigned s_tmp[kScanThreads / 32];
    unsigned v = 0;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
        const unsigned long long t = static_cast<unsigned long long>(blockIdx.x) * kScanTiles + k * kScanThreads + threadIdx.x;
        if (t < tiles) v += counts[t * static_cast<size_t>(kTileStride)];
    }
    unsigned total;
    block_excl_scan<kScanThreads>(v, s_tmp, total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// Ranges, first free positions (cursor) and, for lists of more than kTileChunk pairs, the list of
// chunks. Flags a frame whose pairs exceed the capacity.
__global__ void __launch_bounds__(kScanThreads) tile_scan_kernel(const unsigned* __restrict__ counts, unsigned tiles,
                                                                 const unsigned* __restrict__ sums,
                                                                 uint2* __restrict__ ranges,
                                                                 unsigned* __restrict__ cursor,
                                                                 uint2* __restrict__ chunks, unsigned chunk_cap,
                                                                 unsigned capacity, Ctrl* ctrl) {
    chain_entry();
    __shared__ unsigned s_tmp[kScanThreads / 32];
    const unsigned long long t0 = static_cast<unsigned long long>(blockIdx.x) * kScanTiles + threadIdx.x * kScanPer;
    // The preprocess's total counts whole rectangles, so the pairs to sort are at most as many, and
    // within the capacity every sum fits 32 bits.
    const bool over = ctrl->pair_total > capacity;
    unsigned cnt[kScanPer], own = 0, before = 0;
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) cnt[k] = t0 + k < tiles ? counts[(t0 + k) * kTileStride] : 0u;
    if (over) {
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&ctrl->flags, kFlagOverflow);
        return;
    }
    if (sums) {
        for (unsigned b = threadIdx.x; b < blockIdx.x; b += kScanThreads) before += sums[b];
    } else {
        const unsigned end = blockIdx.x * kScanTiles;
#pragma unroll 4
        for (unsigned t = threadIdx.x; t < end; t += kScanThreads) before += counts[t * static_cast<size_t>(kTileStride)];
    }
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) own += cnt[k];
    unsigned all;
    if (blockIdx.x) {
        block_excl_scan<kScanThreads>(before, s_tmp, all);
        before = all;
    }
    unsigned start = before + block_excl_scan<kScanThreads>(own, s_tmp, all);
#pragma unroll
    for (int k = 0; k < kScanPer; ++k) {
        if (t0 + k >= tiles) break;
        ranges[t0 + k] = cnt[k] ? make_uint2(start, start + cnt[k]) : make_uint2(0u, 0u);
        cursor[(t0 + k) * kTileStride] = start;
        start += cnt[k];
        if (cnt[k] > kTileChunk) {
            const unsigned n = (cnt[k] + kTileChunk - 1) / kTileChunk;
            const unsigned at = atomicAdd(&ctrl->chunk_count, n);
            for (unsigned c = 0; c < n && at + c < chunk_cap; ++c)
                chunks[at + c] = make_uint2(static_cast<unsigned>(t0 + k), c);
        }
    }
}

// ---- scatter -------------------------------------------------------------------------------------

constexpr unsigned kScatterLanes = 32, kScatterFewLanes = 8;  // entries per warp and round, and in a small frame
constexpr unsigned kFewEntries = 1u << 21;  // up to here a warp keeps four pairs per lane in flight, above it two
// Up to here a warp takes 8 entries at a time, above it 32: with 32 a frame of so few entries does not give
// every SM a CTA (20k splats of 800 tiles each, 1920x1080: 240 us of scatter; the frame 611 -> 480 us).
constexpr unsigned kFewestEntries = 148 * kThreads;
constexpr unsigned kLargeArea = 1024;  // an entry of more tiles is left to the whole CTA

// Tile k of a rectangle w tiles wide with corner tile org, in a view of tx tiles per row.
__device__ __forceinline__ unsigned tile_of(unsigned k, unsigned org, unsigned w, unsigned tx) {
    const unsigned row = k / w;
    return org + row * tx + (k - row * w);
}

// Every visible entry's pairs into its tiles' lists. A warp takes 32 entries at a time and spreads
// their pairs over its lanes (a search in the running sum of the rectangles' areas), so that a lane
// holds kScatterPairs appends in flight whatever the rectangles' sizes; entries of more than
// kLargeArea tiles go to the whole CTA afterwards. offs (training; else NULL) receives each
// entry's first gradient slot, allocated per CTA and round in any order.
// kScatterPairs: four where the frame is short of warps and waits for the adds, two in a large frame,
// whose instructions count (a warp's 32 entries have 43 to 69 pairs in the views measured): 191 against
// 193 us per 740k frame, but 6.25 against 6.00 ms for the 64-view batch; equal at 2.2M entries.
// (Spreading the pairs of a CTA's 256 to 1024 entries over its threads takes a fifth of the instructions
// and is no faster; nor is ranking small entries' pairs as they are counted, which saves the scatter
// four fifths of its adds: the scattered accesses themselves bound it.)
template <int kScatterPairs, unsigned kLanes>
__global__ void __launch_bounds__(kThreads) tile_scatter_kernel(const unsigned* __restrict__ depth_key,
                                                                const unsigned long long* __restrict__ rect16,
                                                                unsigned entries, BatchTables tables,
                                                                unsigned* __restrict__ cursor,
                                                                unsigned long long* __restrict__ pairs,
                                                                unsigned* __restrict__ offs, Ctrl* ctrl) {
    chain_entry();
    __shared__ unsigned s_total[kWarps];
    __shared__ unsigned s_base;
    constexpr unsigned kScatterEntries = kLanes * kWarps;  // per CTA and round
    __shared__ unsigned s_large[kScatterEntries];
    __shared__ unsigned s_large_count;
    if (ctrl->flags & kFlagOverflow) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned rounds = entries / kScatterEntries + (entries % kScatterEntries != 0);
    for (unsigned round = blockIdx.x; round < rounds; round += gridDim.x) {
        const unsigned first = round * kScatterEntries + warp * kLanes, e = first + lane;
        if (tid == 0) s_large_count = 0;
        const unsigned key = lane < kLanes && e < entries ? depth_key[e] : kCulledKey;
        const bool visible = key != kCulledKey;
        unsigned org = 0, width = 1, tx = 0, area = 0;
        if (visible) {
            const unsigned long long r = rect16[e];
            const unsigned x0 = r & 0xFFFFu, y0 = (r >> 16) & 0xFFFFu, x1 = (r >> 32) & 0xFFFFu,
                           y1 = static_cast<unsigned>(r >> 48);
            const unsigned v = find_segment(tables.entry_base, tables.n_views, e);
            tx = tables.tiles_x[v];
            org = tables.tile_base[v] + y0 * tx + x0;
            width = x1 - x0 + 1;  // 0 where the bounds are empty
            area = width * (y1 - y0 + 1);
            width = max(width, 1u);
        }
        if (offs) {
            const unsigned incl = warp_incl_scan(area);
            if (lane == 31) s_total[warp] = incl;
            __syncthreads();
            if (tid == 0) {
                unsigned sum = 0;
                for (int w = 0; w < kWarps; ++w) {
                    const unsigned t = s_total[w];
                    s_total[w] = sum;
                    sum += t;
                }
                s_base = sum ? atomicAdd(&ctrl->slot_count, sum) : 0u;
            }
            __syncthreads();
            if (visible) offs[e] = s_base + s_total[warp] + incl - area;
        } else {
            __syncthreads();  // s_large_count
        }
        {
            const bool large = area > kLargeArea;
            if (large) s_large[atomicAdd(&s_large_count, 1u)] = static_cast<unsigned>(warp * kLanes + lane);
            const unsigned spread = large ? 0u : area;
            const unsigned incl = warp_incl_scan(spread);
            const unsigned excl = incl - spread, total = __shfl_sync(0xFFFFFFFFu, incl, 31);
            for (unsigned p0 = 0; p0 < total; p0 += 32 * kScatterPairs) {
                unsigned tile[kScatterPairs], own[kScatterPairs];
#pragma unroll
                for (int u = 0; u < kScatterPairs; ++u) {
                    const unsigned p = p0 + u * 32 + lane;
                    int owner = 0;  // the last lane whose first pair is <= p among those with pairs
#pragma unroll
                    for (int step = 16; step > 0; step >>= 1) {
                        const unsigned f = __shfl_sync(0xFFFFFFFFu, excl, owner + step);
                        if (f <= p) owner += step;
                    }
                    own[u] = static_cast<unsigned>(owner);
                    const unsigned k = p - __shfl_sync(0xFFFFFFFFu, excl, owner);
                    const unsigned o = __shfl_sync(0xFFFFFFFFu, org, owner), w = __shfl_sync(0xFFFFFFFFu, width, owner),
                                   t = __shfl_sync(0xFFFFFFFFu, tx, owner);
                    tile[u] = tile_of(k, o, w, t);
                }
                unsigned pos[kScatterPairs];
#pragma unroll
                for (int u = 0; u < kScatterPairs; ++u)
                    if (p0 + u * 32 + lane < total) pos[u] = atomicAdd(&cursor[tile[u] * static_cast<size_t>(kTileStride)], 1u);
#pragma unroll
                for (int u = 0; u < kScatterPairs; ++u) {
                    const unsigned k = __shfl_sync(0xFFFFFFFFu, key, own[u]);
                    if (p0 + u * 32 + lane < total)
                        pairs[pos[u]] = static_cast<unsigned long long>(k) << 32 | (first + own[u]);
                }
            }
        }
        __syncthreads();
        for (unsigned i = 0; i < s_large_count; ++i) {
            const unsigned e = round * kScatterEntries + s_large[i];
            const unsigned long long r = rect16[e];
            const unsigned long long k32 = static_cast<unsigned long long>(depth_key[e]) << 32 | e;
            const unsigned v = find_segment(tables.entry_base, tables.n_views, e);
            const unsigned x0 = r & 0xFFFFu, y0 = (r >> 16) & 0xFFFFu, x1 = (r >> 32) & 0xFFFFu,
                           y1 = static_cast<unsigned>(r >> 48);
            const unsigned w = x1 - x0 + 1, n = w * (y1 - y0 + 1), tx = tables.tiles_x[v];
            const unsigned org = tables.tile_base[v] + y0 * tx + x0;
            for (unsigned p0 = 0; p0 < n; p0 += kThreads * kScatterPairs) {
                unsigned pos[kScatterPairs];
#pragma unroll
                for (int u = 0; u < kScatterPairs; ++u) {
                    const unsigned p = p0 + u * kThreads + tid;
                    if (p < n) pos[u] = atomicAdd(&cursor[tile_of(p, org, w, tx) * static_cast<size_t>(kTileStride)], 1u);
                }
#pragma unroll
                for (int u = 0; u < kScatterPairs; ++u)
                    if (p0 + u * kThreads + tid < n) pairs[pos[u]] = k32;
            }
        }
        __syncthreads();
    }
}

// ---- sort ----------------------------------------------------------------------------------------

constexpr int kItems = 8;  // pairs per thread
static_assert(kThreads * kItems == kTileChunk, "a chunk is what one CTA sorts");
constexpr unsigned long long kNoPair = ~0ull;  // sorts behind every pair (a culled key never makes one)
constexpr int kBuckets = 512;
constexpr int kBucketsPer = kBuckets / kThreads;
constexpr unsigned kBucketMax = 48;  // a fuller bucket sends the chunk to the merge sort

// Shared-memory place of item i of the merge sort: one word of padding per eight, so that a thread's
// eight consecutive items start in another bank pair than its neighbours'.
__device__ __forceinline__ unsigned padded(unsigned i) { return i + (i >> 3); }

struct SortShared {
    unsigned long long pair[kTileChunk + kTileChunk / 8];
    unsigned start[kBuckets];
    unsigned tmp[kWarps], low[kWarps], high[kWarps];
};

__device__ __forceinline__ void order(unsigned long long& a, unsigned long long& b) {
    const unsigned long long lo = a < b ? a : b, hi = a < b ? b : a;
    a = lo;
    b = hi;
}

// Eight items in registers: Batcher's odd-even merge network (19 exchanges).
__device__ __forceinline__ void sort8(unsigned long long (&v)[kItems]) {
    order(v[0], v[1]); order(v[2], v[3]); order(v[4], v[5]); order(v[6], v[7]);
    order(v[0], v[2]); order(v[1], v[3]); order(v[4], v[6]); order(v[5], v[7]);
    order(v[1], v[2]); order(v[5], v[6]);
    order(v[0], v[4]); order(v[1], v[5]); order(v[2], v[6]); order(v[3], v[7]);
    order(v[2], v[4]); order(v[3], v[5]);
    order(v[1], v[2]); order(v[3], v[4]); order(v[5], v[6]);
}

// The merge sort of the CTA's n (1..kTileChunk) pairs at src; emit(i, pair) receives the i-th. Eight
// pairs per thread in registers, then runs of 8, 16, ... merged pairwise, each thread finding its
// eight outputs by a merge-path search. Merges of up to 256 pairs stay within a warp and need no
// block barrier. Only the threads that n needs take part.
template <typename F>
__device__ __forceinline__ void merge_sort_chunk(const unsigned long long* src, unsigned n, SortShared& sh,
                                                 F&& emit) {
    unsigned long long* s_pair = sh.pair;
    const unsigned tid = threadIdx.x;
    const unsigned need = (n + kItems - 1) / kItems;  // threads with items
    const unsigned total = need * kItems;             // padded with kNoPair
    const bool active = tid < need;
    unsigned long long v[kItems];
    if (active) {
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            const unsigned i = k * need + tid;  // any order will do: neighbouring threads read neighbours
            v[k] = i < n ? src[i] : kNoPair;
        }
        sort8(v);
    }
    for (unsigned run = kItems; run < total; run *= 2) {
        const bool in_warp = 2 * run <= 32 * kItems;
        if (active)
#pragma unroll
            for (int k = 0; k < kItems; ++k) s_pair[padded(tid * kItems + k)] = v[k];
        if (in_warp) __syncwarp();
        else __syncthreads();
        if (active) {
            const unsigned base = tid * kItems / (2 * run) * (2 * run), diag = tid * kItems - base;
            const unsigned la = min(run, total - base), lb = min(run, total - base - la);
            unsigned lo = diag > lb ? diag - lb : 0u, hi = min(diag, la);
            while (lo < hi) {  // items of the first run among the first diag outputs
                const unsigned mid = (lo + hi) >> 1;
                if (s_pair[padded(base + mid)] < s_pair[padded(base + run + diag - 1 - mid)]) lo = mid + 1;
                else hi = mid;
            }
            unsigned a = base + lo, b = base + run + diag - lo;
            const unsigned ea = base + la, eb = base + run + lb;
            unsigned long long va = a < ea ? s_pair[padded(a)] : kNoPair;
            unsigned long long vb = b < eb ? s_pair[padded(b)] : kNoPair;
#pragma unroll
            for (int k = 0; k < kItems; ++k) {
                const bool first = va < vb || b >= eb;
                v[k] = first ? va : vb;
                a += first;
                b += !first;
                const unsigned p = first ? a : b, e = first ? ea : eb;
                const unsigned long long next = p < e ? s_pair[padded(p)] : kNoPair;
                va = first ? next : va;
                vb = first ? vb : next;
            }
        }
        if (in_warp) __syncwarp();
        else __syncthreads();
    }
    if (active)
#pragma unroll
        for (int k = 0; k < kItems; ++k) s_pair[padded(tid * kItems + k)] = v[k];
    __syncthreads();
    for (unsigned i = tid; i < n; i += kThreads) emit(i, s_pair[padded(i)]);
}

// Sorts the CTA's n (1..kTileChunk) pairs at src; emit(i, pair) receives the i-th. The pairs are
// distributed over kBuckets equal steps between the chunk's smallest and largest depth key, and each
// pair's place is its bucket's start plus the number of smaller pairs in its bucket: a bucket holds
// one or two, so that costs a few compares where a merge sort takes nine merge levels. A chunk whose
// depths crowd into a few buckets (more than kBucketMax pairs in one) is merge-sorted.
template <typename F>
__device__ __forceinline__ void sort_chunk(const unsigned long long* src, unsigned n, SortShared& sh, F&& emit) {
    const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned low = 0xFFFFFFFFu, high = 0;
#pragma unroll
    for (int k = 0; k < kBucketsPer; ++k) sh.start[k * kThreads + tid] = 0;
    for (unsigned i = tid; i < n; i += kThreads) {
        const unsigned key = static_cast<unsigned>(src[i] >> 32);
        low = min(low, key);
        high = max(high, key);
    }
    low = __reduce_min_sync(0xFFFFFFFFu, low);
    high = __reduce_max_sync(0xFFFFFFFFu, high);
    if (lane == 0) {
        sh.low[warp] = low;
        sh.high[warp] = high;
    }
    __syncthreads();
    low = __reduce_min_sync(0xFFFFFFFFu, sh.low[lane & (kWarps - 1)]);
    high = __reduce_max_sync(0xFFFFFFFFu, sh.high[lane & (kWarps - 1)]);
    // Monotone in the key: conversion, product and truncation each are.
    const float scale = static_cast<float>(kBuckets) / (static_cast<float>(high - low) + 1.0f);
    const auto bucket_of = [&](unsigned long long x) {
        const unsigned b = static_cast<unsigned>(static_cast<float>(static_cast<unsigned>(x >> 32) - low) * scale);
        return min(b, static_cast<unsigned>(kBuckets - 1));
    };
    for (unsigned i = tid; i < n; i += kThreads) atomicAdd(&sh.start[bucket_of(src[i])], 1u);
    __syncthreads();
    unsigned cnt[kBucketsPer], own = 0, most = 0;
#pragma unroll
    for (int k = 0; k < kBucketsPer; ++k) {
        cnt[k] = sh.start[tid * kBucketsPer + k];
        own += cnt[k];
        most = max(most, cnt[k]);
    }
    if (__syncthreads_or(most > kBucketMax)) {
        merge_sort_chunk(src, n, sh, emit);
        return;
    }
    unsigned all;
    unsigned start = block_excl_scan<kThreads>(own, sh.tmp, all);
#pragma unroll
    for (int k = 0; k < kBucketsPer; ++k) {
        sh.start[tid * kBucketsPer + k] = start;
        start += cnt[k];
    }
    __syncthreads();
    // Into the buckets; afterwards a bucket's start has become its end, the next one's start.
    for (unsigned i = tid; i < n; i += kThreads) {
        const unsigned long long x = src[i];
        sh.pair[atomicAdd(&sh.start[bucket_of(x)], 1u)] = x;
    }
    __syncthreads();
    // In bucket order, so that neighbouring threads emit neighbouring places.
    for (unsigned i = tid; i < n; i += kThreads) {
        const unsigned long long x = sh.pair[i];
        const unsigned b = bucket_of(x);
        const unsigned s0 = b ? sh.start[b - 1] : 0u, s1 = sh.start[b];
        unsigned place = s0;
        for (unsigned j = s0; j < s1; ++j) place += sh.pair[j] < x;
        emit(place, x);
    }
}

// One warp's sort of n (0..kShortList) pairs at src into entries at out, two pairs per lane: a pair's place
// is the number of smaller ones, counted as the warp passes every pair round.
constexpr unsigned kShortList = 64;
__device__ __forceinline__ void sort_short(const unsigned long long* src, unsigned n, unsigned* out) {
    const unsigned lane = threadIdx.x & 31;
    const unsigned long long x0 = lane < n ? src[lane] : kNoPair, x1 = lane + 32 < n ? src[lane + 32] : kNoPair;
    unsigned place0 = 0, place1 = 0;
    for (unsigned j = 0; j < min(n, 32u); ++j) {
        const unsigned long long x = __shfl_sync(0xFFFFFFFFu, x0, j);
        place0 += x < x0;
        place1 += x < x1;
    }
    for (unsigned j = 32; j < n; ++j) {
        const unsigned long long x = __shfl_sync(0xFFFFFFFFu, x1, j - 32);
        place0 += x < x0;
        place1 += x < x1;
    }
    if (lane < n) out[place0] = static_cast<unsigned>(x0);
    if (lane + 32 < n) out[place1] = static_cast<unsigned>(x1);
}

// CTA b < tiles sorts tile b's first chunk, the others take the further chunks of long lists in turn.
// A list of one chunk is written as sorted entries; a chunk of a longer one goes back in place.
// Latency-bound: eight CTAs per SM (32 registers, where only the merge sort spills) instead of five take
// 192 to 189 us off the 740k frame, 403 to 396 us at 2.2M / 1920x1080, 2.29 to 2.22 ms off 16 views. Crowded
// depths (the merge sort) cost little: a wall of 740k splats takes 271 us a frame, a plane 277 us (with the
// LSD chain 365 and 503 us). Chunks of 1024 in CTAs of 128 threads: 392 us and 2.19 ms, but the lists of
// small images then need merging (the 64-view batch 6.15 against 5.92 ms).
//
// A list of at most kShortList pairs is sorted by one warp. Where a frame has few entries for its tiles
// (kSparse), most lists are that short or empty, and a CTA takes eight tiles, a warp each, and then their
// longer lists one after another: ten 572x327 views of
// 32k Gaussians in 8x8 tiles take 295 us a frame with a CTA's sort for every list, 238 with the warp's,
// 214 with eight tiles per CTA; eight 1660x984 views of two scenes of 20k in 16x32 tiles 269, 242, 230 us.
// With many entries per tile a CTA per tile is the better one: 2.22 against 2.24 ms for 16 views of 740k.
template <bool kSparse>
__global__ void __launch_bounds__(kThreads, 8) tile_sort_kernel(const uint2* __restrict__ ranges, unsigned tiles,
                                                             const uint2* __restrict__ chunks, unsigned chunk_cap,
                                                             unsigned long long* pairs,
                                                             unsigned* __restrict__ vals, const Ctrl* ctrl) {
    chain_entry();
    __shared__ SortShared sh;
    if (ctrl->flags & kFlagOverflow) return;
    constexpr unsigned kTiles = kSparse ? kWarps : 1;  // of a CTA
    const unsigned list_ctas = (tiles + kTiles - 1) / kTiles;
    if (blockIdx.x < list_ctas) {
        const auto sort_list = [&](uint2 r, unsigned n) {
            if (n <= kTileChunk)
                sort_chunk(pairs + r.x, n, sh, [&](unsigned i, unsigned long long x) { vals[r.x + i] = static_cast<unsigned>(x); });
            else
                sort_chunk(pairs + r.x, kTileChunk, sh, [&](unsigned i, unsigned long long x) { pairs[r.x + i] = x; });
        };
        if (!kSparse) {
            const uint2 r = ranges[blockIdx.x];
            const unsigned n = r.y - r.x;
            if (n > kShortList) sort_list(r, n);
            else if (threadIdx.x < 32) sort_short(pairs + r.x, n, vals + r.x);
            return;
        }
        const unsigned first = blockIdx.x * kTiles, end = min(first + kTiles, tiles), mine = first + (threadIdx.x >> 5);
        const uint2 own = mine < end ? ranges[mine] : make_uint2(0u, 0u);
        if (own.y - own.x <= kShortList) sort_short(pairs + own.x, own.y - own.x, vals + own.x);
        if (!__syncthreads_or(own.y - own.x > kShortList)) return;
        for (unsigned t = first; t < end; ++t) {
            const uint2 r = ranges[t];
            const unsigned n = r.y - r.x;
            if (n <= kShortList) continue;
            __syncthreads();
            sort_list(r, n);
        }
        return;
    }
    const unsigned count = min(ctrl->chunk_count, chunk_cap);
    for (unsigned c = blockIdx.x - list_ctas; c < count; c += gridDim.x - list_ctas) {
        const uint2 ch = chunks[c];
        if (ch.y == 0) continue;
        const uint2 r = ranges[ch.x];
        const unsigned at = r.x + ch.y * kTileChunk;
        __syncthreads();
        sort_chunk(pairs + at, min(kTileChunk, r.y - at), sh, [&](unsigned i, unsigned long long x) { pairs[at + i] = x; });
    }
}

// Merges the sorted chunks of every list of several: the place of a pair is its place in its own
// chunk plus, for every other chunk of its group (kTileGroup chunks), the number of smaller pairs there.
// Both chunks lie in shared memory and the CTA merges them, sixteen outputs per thread from a merge-path
// search: each pair of its own is passed once and gets the other chunk's place of the moment. A list of one
// group is written as sorted entries; a group of a longer one as pairs to `merged`, for
// tile_merge_groups_kernel. (With a search of eleven steps for every pair instead, 740k splats
// within 70 pixels take 1026 us a frame, with the merges 914; within 140 pixels 462 and 444; 64 views of 1M
// 5.91 and 5.86 ms.)
__global__ void __launch_bounds__(kThreads) tile_merge_kernel(const uint2* __restrict__ ranges,
                                                              const uint2* __restrict__ chunks, unsigned chunk_cap,
                                                              const unsigned long long* __restrict__ pairs,
                                                              unsigned long long* __restrict__ merged,
                                                              unsigned* __restrict__ vals, const Ctrl* ctrl) {
    chain_entry();
    constexpr unsigned kOutputs = 2 * kItems;  // of two whole chunks, per thread
    __shared__ unsigned long long s_own[kTileChunk + kTileChunk / 8], s_other[kTileChunk + kTileChunk / 8];
    __shared__ unsigned s_place[kTileChunk];
    if (ctrl->flags & kFlagOverflow) return;
    const unsigned count = min(ctrl->chunk_count, chunk_cap);
    for (unsigned c = blockIdx.x; c < count; c += gridDim.x) {
        const uint2 ch = chunks[c];
        const uint2 r = ranges[ch.x];
        const unsigned of = (r.y - r.x + kTileChunk - 1) / kTileChunk;  // chunks of the list
        const unsigned g0 = ch.y / kTileGroup * kTileGroup, g1 = min(of, g0 + kTileGroup);
        const unsigned at = r.x + ch.y * kTileChunk, m = min(kTileChunk, r.y - at);
        __syncthreads();
        for (unsigned i = threadIdx.x; i < m; i += kThreads) {
            s_own[padded(i)] = pairs[at + i];
            s_place[i] = i;
        }
        for (unsigned o = g0; o < g1; ++o) {
            if (o == ch.y) continue;
            const unsigned oat = r.x + o * kTileChunk, om = min(kTileChunk, r.y - oat);
            __syncthreads();
            for (unsigned i = threadIdx.x; i < om; i += kThreads) s_other[padded(i)] = pairs[oat + i];
            __syncthreads();
            const unsigned diag = threadIdx.x * kOutputs;
            if (diag >= m + om) continue;
            unsigned lo = diag > om ? diag - om : 0u, hi = min(diag, m);
            while (lo < hi) {  // own pairs among the first diag outputs
                const unsigned mid = (lo + hi) >> 1;
                if (s_own[padded(mid)] < s_other[padded(diag - 1 - mid)]) lo = mid + 1;
                else hi = mid;
            }
            unsigned a = lo, b = diag - lo;
            unsigned long long va = a < m ? s_own[padded(a)] : kNoPair, vb = b < om ? s_other[padded(b)] : kNoPair;
#pragma unroll
            for (unsigned k = 0; k < kOutputs; ++k) {
                const bool own = va < vb;
                if (own) s_place[a] += b;
                a += own;
                b += !own;
                const unsigned p = own ? a : b, end = own ? m : om;
                const unsigned long long next = p < end ? (own ? s_own : s_other)[padded(p)] : kNoPair;
                va = own ? next : va;
                vb = own ? vb : next;
            }
        }
        __syncthreads();
        const unsigned out = r.x + g0 * kTileChunk;
        for (unsigned i = threadIdx.x; i < m; i += kThreads) {
            const unsigned long long x = s_own[padded(i)];
            if (of <= kTileGroup) vals[out + s_place[i]] = static_cast<unsigned>(x);
            else merged[out + s_place[i]] = x;
        }
    }
}

// Lists of several groups (more than kTileGroup * kTileChunk pairs in one tile): each pair's place is its
// place in its own sorted group plus the number of smaller pairs in every other group of the list.
__global__ void __launch_bounds__(kThreads) tile_merge_groups_kernel(const uint2* __restrict__ ranges,
                                                                     const uint2* __restrict__ chunks,
                                                                     unsigned chunk_cap,
                                                                     const unsigned long long* __restrict__ merged,
                                                                     unsigned* __restrict__ vals, const Ctrl* ctrl) {
    chain_entry();
    if (ctrl->flags & kFlagOverflow) return;
    constexpr unsigned kGroupPairs = kTileGroup * kTileChunk;
    const unsigned count = min(ctrl->chunk_count, chunk_cap);
    for (unsigned c = blockIdx.x; c < count; c += gridDim.x) {
        const uint2 ch = chunks[c];
        const uint2 r = ranges[ch.x];
        if (r.y - r.x <= kGroupPairs) continue;
        const unsigned at = ch.y * kTileChunk, m = min(kTileChunk, r.y - r.x - at);  // within the list
        const unsigned own = ch.y / kTileGroup;
        for (unsigned i = threadIdx.x; i < m; i += kThreads) {
            const unsigned long long x = merged[r.x + at + i];
            unsigned place = at + i - own * kGroupPairs;
            for (unsigned g = 0; g * kGroupPairs < r.y - r.x; ++g) {
                if (g == own) continue;
                const unsigned long long* s = merged + r.x + g * kGroupPairs;
                unsigned lo = 0, hi = min(kGroupPairs, r.y - r.x - g * kGroupPairs);
                while (lo < hi) {
                    const unsigned mid = (lo + hi) >> 1;
                    if (s[mid] < x) lo = mid + 1;
                    else hi = mid;
                }
                place += lo;
            }
            vals[r.x + place] = static_cast<unsigned>(x);
        }
    }
}

unsigned scan_ctas(unsigned tiles) { return std::max(1u, (tiles + kScanTiles - 1) / kScanTiles); }

}  // namespace

size_t tile_count_words(uint64_t tiles) { return static_cast<size_t>(tiles) * kTileStride; }
size_t tile_sum_words(uint64_t tiles) { return static_cast<size_t>((tiles + kScanTiles - 1) / kScanTiles) + 1; }
size_t tile_chunk_entries(uint64_t capacity) { return 2 * static_cast<size_t>(capacity / kTileChunk) + 2; }

void launch_tile_sort(const TileSortArgs& a, cudaStream_t stream) {
    const unsigned ctas = scan_ctas(a.tiles);
    const bool sums = a.tiles > kScanDirect;
    if (sums) launch_chained(tile_sums_kernel, dim3(ctas), dim3(kScanThreads), stream, a.counts, a.tiles, a.sums);
    launch_chained(tile_scan_kernel, dim3(ctas), dim3(kScanThreads), stream, a.counts, a.tiles,
                   sums ? static_cast<const unsigned*>(a.sums) : nullptr, a.ranges, a.cursor, a.chunks, a.chunk_cap,
                   a.capacity, a.ctrl);
    const bool few = a.entries <= kFewestEntries;
    const uint64_t per = (few ? kScatterFewLanes : kScatterLanes) * kWarps;
    const unsigned rounds = static_cast<unsigned>((a.entries + per - 1) / per);
    const auto scatter = few                        ? tile_scatter_kernel<4, kScatterFewLanes>
                         : a.entries <= kFewEntries ? tile_scatter_kernel<4, kScatterLanes>
                                                    : tile_scatter_kernel<2, kScatterLanes>;
    launch_chained(scatter, dim3(std::max(1u, std::min(rounds, 148u * 32u))), dim3(kThreads), stream,
                   a.depth_key, a.rect16, a.entries, a.tables, a.cursor, a.pairs, a.offs, a.ctrl);
    // More in step with the capacity, which grows with the pairs: 296 CTAs left 300k splats of 59 tiles each
    // waiting for their further chunks (556 us a frame, with this and the merge's grid 504).
    const unsigned further = std::min(a.chunk_cap, std::max(296u, std::min(a.chunk_cap / 8, 148u * 8u)));
    const bool sparse = sparse_frame(a.entries, a.tiles);
    const unsigned list_ctas = sparse ? (a.tiles + kWarps - 1) / kWarps : a.tiles;
    launch_chained(sparse ? tile_sort_kernel<true> : tile_sort_kernel<false>, dim3(list_ctas + further), dim3(kThreads),
                   stream, a.ranges, a.tiles, a.chunks, a.chunk_cap, a.pairs, a.vals, a.ctrl);
    if (a.longest <= kTileChunk) return;
    launch_chained(tile_merge_kernel, dim3(std::max(1u, std::min(a.chunk_cap / 2, 148u * 5u))), dim3(kThreads), stream,
                   a.ranges, a.chunks, a.chunk_cap, a.pairs, a.merged, a.vals, a.ctrl);
    if (a.longest <= kTileGroup * kTileChunk) return;
    launch_chained(tile_merge_groups_kernel, dim3(std::min(a.chunk_cap, 592u)), dim3(kThreads), stream, a.ranges,
                   a.chunks, a.chunk_cap, a.merged, a.vals, a.ctrl);
}

}  // namespace ab2
