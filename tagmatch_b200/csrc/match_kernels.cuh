// Device kernels of the batched matcher (routing, slices, subset test, key
// gather, match_unique).  Included by match.cu (the engine's pipeline) and
// noalloc.cu (the pipeline over caller-free static scratch); each
// translation unit gets its own internal copy.
#pragma once
#include <algorithm>
#include <type_traits>
#include "match.cuh"

namespace tmb {
namespace {

constexpr int kMatchThreads = 256;
constexpr int kMatchWarps = kMatchThreads / 32;
constexpr int kWarpRecs = 64;  // staged hit records per warp (1 KB)
static_assert(kItemQueries == 1024, "an item's queries are 32 words of 32, one per lane");
constexpr unsigned long long kSpinLimit = 1ull << 26;

inline unsigned blocks_for(size_t n, unsigned t) { return unsigned((n + t - 1) / t); }

// ---------------------------------------------------------------------------
// Routing
// ---------------------------------------------------------------------------
constexpr int kSliceRows = kBits + 1;  // 192 bit rows + the all-zero padding row
constexpr int kSliceWords = kSliceRows * 8;  // 193 x 256 bits

constexpr int kRouteThreads = 256;        // queries per routing CTA
constexpr uint32_t kRouteParts = 64;      // partition masks per routing CTA
constexpr uint32_t kGroupQueries = 8192;  // queries per count group: 256 words of a partition's routing row
// Queue positions per queue-filling CTA (4 chunks; 20,011 queries on 125
// partitions: 72 us with 2,048 positions, 59 with 1,024, 57 with 512, where
// 65,536 on 382 take 345, 351 and 371).
constexpr uint32_t kFillRanks = 1024;
constexpr int kPlanThreads = 1024;

// Words of one partition's routing row (a bit per query, whole CTAs).
__host__ __device__ inline uint32_t route_row_words(uint32_t nq) { return (nq + kRouteThreads - 1) / kRouteThreads * 8; }
// Count groups per partition (0: the partition's count is enough).
__host__ __device__ inline uint32_t route_groups(uint32_t nq) {
    return nq <= kGroupQueries ? 0u : (nq + kGroupQueries - 1) / kGroupQueries;
}

// Routing matrix of partitions [p0, p1): bit l of rows[p - p0][w] is set when
// partition p's mask is a subset of query 32 w + l.  Lane = query; the masks
// are read from shared memory, one vote per (partition, 32 queries).  COUNT
// adds each partition's queries to part_count (and to the partition's count
// of every kGroupQueries queries), zeroed by the caller.  Queries x
// partitions spread over the grid, so that a few queries or a few
// partitions still make enough CTAs: testing all partitions in one CTA per
// 256 queries, twice, took 500 of the 1,390 us of 4,096 queries on 2,082
// partitions.
template <bool COUNT>
__global__ void __launch_bounds__(kRouteThreads) k_route(const uint32_t *__restrict__ queries, uint32_t nq,
                                                         const uint32_t *__restrict__ part_mask, uint32_t p0, uint32_t p1,
                                                         uint32_t *__restrict__ rows, uint32_t *__restrict__ part_count,
                                                         uint32_t *__restrict__ group_count) {
    __shared__ uint4 s_mask[kRouteParts * 2];
    __shared__ uint32_t s_row[32][kRouteThreads / 32 + 1];
    const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t pb = p0 + blockIdx.y * kRouteParts;
    const uint32_t np = min(kRouteParts, p1 - pb);
    const uint4 *masks = reinterpret_cast<const uint4 *>(part_mask);
    for (uint32_t i = tid; i < 2 * np; i += kRouteThreads) s_mask[i] = masks[size_t(pb) * 2 + i];
    const uint32_t qi = blockIdx.x * kRouteThreads + tid;
    uint32_t q[kWords];
#pragma unroll
    for (int k = 0; k < kWords; ++k) q[k] = qi < nq ? queries[size_t(qi) * kWords + k] : 0u;
    const uint32_t live = __ballot_sync(kFull, qi < nq);
    const uint32_t row_words = route_row_words(nq), groups = route_groups(nq);
    __syncthreads();
    for (uint32_t b = 0; b < np; b += 32) {
        uint32_t mine = 0;  // partition pb + b + lane: the warp's queries
        const uint32_t nb = min(32u, np - b);
        for (uint32_t i = 0; i < nb; ++i) {
            const uint4 m0 = s_mask[2 * (b + i)], m1 = s_mask[2 * (b + i) + 1];
            uint32_t x = m0.x & ~q[0];
            x = andnot_or(m0.y, q[1], x);
            x = andnot_or(m0.z, q[2], x);
            x = andnot_or(m0.w, q[3], x);
            x = andnot_or(m1.x, q[4], x);
            x = andnot_or(m1.y, q[5], x);
            const uint32_t hit = __ballot_sync(kFull, x == 0);
            if (lane == i) mine = hit;
        }
        s_row[lane][warp] = mine & live;
        __syncthreads();
        // eight threads per partition write its 256 queries' words
        const uint32_t r = tid >> 3, w = tid & 7, p = pb + b + r;
        const uint32_t word = s_row[r][w];
        if (r < nb) rows[size_t(p - p0) * row_words + blockIdx.x * 8 + w] = word;
        if (COUNT) {
            uint32_t c = __popc(word);
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) c += __shfl_xor_sync(kFull, c, o);
            if (w == 0 && r < nb && c) {
                atomicAdd(&part_count[p], c);
                if (groups) atomicAdd(&group_count[size_t(p) * groups + blockIdx.x * kRouteThreads / kGroupQueries], c);
            }
        }
        __syncthreads();
    }
}

// Tiles per work item of a batch: the configured number, halved until the
// batch has kItemsPerCta items for each of the subset test's CTAs, or an item
// would no longer give its eight warps a step of tiles each.  With fewer items
// than that a batch takes as long as its largest item: 1,000 queries on a
// million filters make 312 items of 128 tiles for 592 CTAs.  Measured
// there and with 2,000 queries on 300,000 (us): as configured 374 and 512,
// with 2 items per CTA 322 and 428, with 4 309 and 430; with 8 the claims cost
// what they even out.
constexpr uint32_t kItemsPerCta = 4;
constexpr int kSegHalvings = 5;
__host__ __device__ inline uint32_t least_seg(uint32_t nq) {
    uint32_t tiles = 32;  // a warp's tiles per step, for items of nq queries
    for (uint32_t words = (nq + 31) / 32; tiles > 1 && words > 1; words = (words + 1) / 2) tiles /= 2;
    return kMatchWarps * tiles;
}
__host__ __device__ inline uint32_t halved_seg(uint32_t seg, int halvings, uint32_t least) {
    const uint32_t s = seg >> halvings;
    return s > least ? s : seg < least ? seg : least;
}
// Work items of a partition with `count` queries and nt tiles.
__host__ __device__ inline uint32_t part_items(uint32_t count, uint32_t nt, uint32_t seg) {
    return (count + kItemQueries - 1) / kItemQueries * ((nt + seg - 1) / seg);
}

// Offsets of the work plan from the partitions' counts, one CTA: queue
// positions, 256-query chunks, and work items (groups of kItemChunks chunks
// x tile segments), the items over queue positions (order: the partition at
// each position; null: id order).  seg_out: tiles per item, from seg_tiles
// and the items wanted (0: seg_tiles as it is); queue positions; chunks.
__global__ void __launch_bounds__(kPlanThreads) k_plan(const uint32_t *__restrict__ part_count,
                                                       const uint32_t *__restrict__ part_tile_begin,
                                                       const uint32_t *__restrict__ order, uint32_t n_parts,
                                                       uint32_t seg_tiles, uint32_t least, uint32_t want_items,
                                                       uint32_t *__restrict__ part_off, uint32_t *__restrict__ chunk_off,
                                                       uint32_t *__restrict__ item_off, uint32_t *__restrict__ seg_out) {
    __shared__ uint32_t s_sum[3][kPlanThreads / 32];
    __shared__ uint32_t s_items[kSegHalvings];  // items are counted in 32 bits
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t seg = seg_tiles;
    if (want_items) {
        if (threadIdx.x < kSegHalvings) s_items[threadIdx.x] = 0;
        __syncthreads();
        uint32_t items[kSegHalvings] = {};
        for (uint32_t p = threadIdx.x; p < n_parts; p += kPlanThreads) {
            const uint32_t count = part_count[p], nt = part_tile_begin[p + 1] - part_tile_begin[p];
#pragma unroll
            for (int h = 0; h < kSegHalvings; ++h) items[h] += part_items(count, nt, halved_seg(seg_tiles, h, least));
        }
#pragma unroll
        for (int h = 0; h < kSegHalvings; ++h) {
            const uint32_t sum = __reduce_add_sync(kFull, items[h]);
            if (lane == 0 && sum) atomicAdd(&s_items[h], sum);
        }
        __syncthreads();
        for (int h = 0; h < kSegHalvings && s_items[h] < want_items; ++h) seg = halved_seg(seg_tiles, h + 1, least);
    }
    uint32_t base[3] = {0, 0, 0};
    for (uint32_t t0 = 0; t0 < n_parts; t0 += kPlanThreads) {
        const uint32_t pos = t0 + threadIdx.x;
        uint32_t v[3] = {0, 0, 0};
        if (pos < n_parts) {
            v[0] = part_count[pos];
            v[1] = (v[0] + kChunk - 1) / kChunk;
            const uint32_t p = order ? order[pos] : pos;
            v[2] = part_items(part_count[p], part_tile_begin[p + 1] - part_tile_begin[p], seg);
        }
        uint32_t incl[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            incl[k] = warp_incl_scan(v[k]);
            if (lane == 31) s_sum[k][warp] = incl[k];
        }
        __syncthreads();
        if (warp < 3) s_sum[warp][lane] = warp_incl_scan(s_sum[warp][lane]);
        __syncthreads();
        uint32_t *out[3] = {part_off, chunk_off, item_off};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if (pos < n_parts) out[k][pos] = base[k] + (warp ? s_sum[k][warp - 1] : 0u) + incl[k] - v[k];
            base[k] += s_sum[k][kPlanThreads / 32 - 1];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part_off[n_parts] = base[0];
        chunk_off[n_parts] = base[1];
        item_off[n_parts] = base[2];
        seg_out[0] = seg;
        seg_out[1] = base[0];
        seg_out[2] = base[1];
    }
}

// Fills the partitions' queues from their routing rows (partitions
// [p0, p0 + gridDim.x)): CTA (p, y) takes the queries of positions
// [1024 y, 1024 y + 1024), finds them in the row (counts per group, then a
// prefix sum over a group's words), and per 256-query chunk writes the queue
// records (words 0 .. 3 in one plane; words 4 and 5, the query id and a pad
// in the other) and the chunk's bit-sliced masks: z[b * 8 + w] bit l is set when query 32 w + l of the chunk
// lacks filter bit b, or does not exist (so an absent query is never a
// candidate).  The slices are bit transposes of the query words, 15
// instructions per 32 x 32 bits where a vote per bit took 128; they leave
// through shared memory (words swizzled over the banks) in whole lines.
__global__ void __launch_bounds__(kChunk) k_fill_queues(const uint32_t *__restrict__ queries, uint32_t nq,
                                                        const uint32_t *__restrict__ rows, uint32_t p0,
                                                        const uint32_t *__restrict__ part_count,
                                                        const uint32_t *__restrict__ group_count,
                                                        const uint32_t *__restrict__ part_off,
                                                        const uint32_t *__restrict__ chunk_off,
                                                        uint4 *__restrict__ queue_lo, uint4 *__restrict__ queue_hi,
                                                        uint32_t *__restrict__ slices) {
    static_assert(kScanThreads == kChunk && kGroupQueries == 32 * kChunk, "one routing word per thread and group");
    __shared__ uint32_t s_list[kFillRanks];
    __shared__ uint32_t s_z[kSliceWords];
    const uint32_t p = p0 + blockIdx.x, r0 = blockIdx.y * kFillRanks, count = part_count[p];
    if (r0 >= count) return;
    const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t r1 = min(count, r0 + kFillRanks);
    const uint32_t row_words = route_row_words(nq), groups = route_groups(nq);
    const uint32_t *row = rows + size_t(blockIdx.x) * row_words;
    uint32_t at = 0;  // position of the group's first query
    for (uint32_t w0 = 0, g = 0; w0 < row_words && at < r1; w0 += kChunk, ++g) {
        const uint32_t in_group = groups ? group_count[size_t(p) * groups + g] : count;
        if (at + in_group > r0) {
            uint32_t x = w0 + tid < row_words ? row[w0 + tid] : 0u;
            uint32_t total;
            uint32_t r = at + block_excl_scan<uint32_t>(__popc(x), total);
            for (; x && r < r1; ++r) {
                if (r >= r0) s_list[r - r0] = (w0 + tid) * 32 + __ffs(x) - 1;
                x &= x - 1;
            }
        }
        at += in_group;
    }
    __syncthreads();
    const uint32_t qbase = part_off[p] + r0, c0 = chunk_off[p] + r0 / kChunk;
    for (uint32_t j0 = 0; r0 + j0 < r1; j0 += kChunk) {
        const uint32_t j = j0 + tid;
        uint32_t q[kWords] = {0, 0, 0, 0, 0, 0};
        if (r0 + j < r1) {
            const uint32_t qi = s_list[j];
#pragma unroll
            for (int k = 0; k < kWords; ++k) q[k] = queries[size_t(qi) * kWords + k];
            queue_lo[size_t(qbase) + j] = make_uint4(q[0], q[1], q[2], q[3]);
            queue_hi[size_t(qbase) + j] = make_uint4(q[4], q[5], qi, 0u);
        }
#pragma unroll
        for (int k = 0; k < kWords; ++k) {
            const uint32_t row_z = k * 32 + lane;
            s_z[row_z * 8 + (warp ^ ((row_z >> 2) & 7))] = ~warp_transpose(q[k], lane);
        }
        if (tid < 8) s_z[kNoBit * 8 + tid] = 0u;  // the padding row: no query lacks it
        __syncthreads();
        uint32_t *zc = slices + size_t(c0 + j0 / kChunk) * kSliceWords;
        for (uint32_t i = tid; i < uint32_t(kSliceWords); i += kChunk)
            zc[i] = s_z[i < kNoBit * 8 ? (i & ~7u) + ((i ^ (i >> 5)) & 7u) : i];
        __syncthreads();
    }
}

// Partitions per routing window, and windows: a window's rows take at most
// `words` words.
inline uint32_t route_window(uint32_t n_parts, uint32_t nq, size_t words) {
    const size_t fit = words / route_row_words(nq) / 32 * 32;
    return uint32_t(std::min<size_t>(n_parts, std::max<size_t>(fit, 32)));
}

// Routing rows of partitions [p0, p1), counted or not.
inline void launch_route(bool count, const uint32_t *d_queries, uint32_t nq, const DevTable &t, uint32_t p0, uint32_t p1,
                         uint32_t *rows, uint32_t *part_count, uint32_t *group_count, cudaStream_t st) {
    const dim3 grid(blocks_for(nq, kRouteThreads), blocks_for(p1 - p0, kRouteParts));
    if (count) k_route<true><<<grid, kRouteThreads, 0, st>>>(d_queries, nq, t.part_mask.p, p0, p1, rows, part_count, group_count);
    else k_route<false><<<grid, kRouteThreads, 0, st>>>(d_queries, nq, t.part_mask.p, p0, p1, rows, part_count, group_count);
    TM_CHECK_LAUNCH();
}

// Queues and slices of every partition, a window of routing rows at a time.
// rows holds the only window's rows already, or each window's are made again.
inline void launch_fill_queues(const uint32_t *d_queries, uint32_t nq, const DevTable &t, uint32_t window, uint32_t *rows,
                               uint32_t *part_count, uint32_t *group_count, const uint32_t *part_off,
                               const uint32_t *chunk_off, uint4 *queue_lo, uint4 *queue_hi, uint32_t *slices, cudaStream_t st) {
    for (uint32_t p0 = 0; p0 < t.n_parts; p0 += window) {
        const uint32_t p1 = std::min(t.n_parts, p0 + window);
        if (window < t.n_parts) launch_route(false, d_queries, nq, t, p0, p1, rows, part_count, group_count, st);
        k_fill_queues<<<dim3(p1 - p0, blocks_for(nq, kFillRanks)), kChunk, 0, st>>>(
            d_queries, nq, rows, p0, part_count, group_count, part_off, chunk_off, queue_lo, queue_hi, slices);
        TM_CHECK_LAUNCH();
    }
}

// ---------------------------------------------------------------------------
// Matching
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// One bulk (non-tensor, non-multicast) TMA copy global -> shared memory.
__device__ __forceinline__ void tma_bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Bounded wait on an mbarrier phase; false when the limit expired.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
    unsigned long long spins = 0;
    while (!mbar_try_wait(bar, parity)) {
        if (++spins > kSpinLimit) return false;
    }
    return true;
}

// Keys of the filters in a hit mask.  The table keeps keys in slot order, so
// a run of adjacent set bits [lo, hi) is the one key range [o[lo], o[hi])
// (o: the tile's slot key offsets, 33 of them).  Calls f(begin, end) per run.
template <class F>
__device__ __forceinline__ void for_each_key_run(const uint32_t *__restrict__ o, uint32_t mask, F f) {
    uint64_t m = mask;
    while (m) {
        const int lo = __ffsll(m) - 1;
        const uint64_t filled = m + (1ull << lo);  // the carry clears the run and sets bit hi
        const int hi = __ffsll(filled & ~m) - 1;
        f(o[lo], o[hi]);
        m &= filled;
    }
}

// Keys of hit mask m of tile t: from the tile's key-count bit planes, or,
// when m touches a filter with 8 keys or more, from the slot offsets.
__device__ __forceinline__ uint32_t mask_keys(const TileKeys &tk, uint32_t m, const uint32_t *__restrict__ slot_key_off,
                                              uint32_t t) {
    if (!(m & tk.wide)) return keys_of_mask(tk, m);
    uint32_t nk = 0;
    for_each_key_run(slot_key_off + size_t(t) * kTile, m, [&](uint32_t b, uint32_t e) { nk += e - b; });
    return nk;
}

struct MatchArgs {
    const uint32_t *tile_words;
    const TileInfo *tile_info;
    const TileKeys *tile_keys;
    const uint32_t *slot_key_off;
    const uint32_t *part_tile_begin;
    const uint32_t *part_count;
    const uint32_t *part_off;
    const uint32_t *item_off;
    const uint32_t *chunk_off;
    const uint4 *queue_lo, *queue_hi;
    const uint32_t *slices;
    uint32_t n_parts;
    const uint32_t *seg;           // tiles per work item (k_plan)
    // [0] next item, [1] hit records, [2] error flags, [3] matching
    // (query, filter) pairs
    unsigned long long *counters;
    HitRec *recs;
    unsigned long long rec_cap;
    uint32_t *qkeys;               // [batch queries] key totals, zeroed by the caller
    uint32_t fpl_trip_cost;        // path choice: estimated cost of one 4-candidate trip of the lane-per-filter loop
    // work-queue order: item_off runs over positions, part_order[pos] is the
    // partition at that position (null: partition id order)
    const uint32_t *part_order;
    // optional timing record per item: [2 item] warp-cycles summed over the
    // CTA's warps, [2 item + 1] hit records; null when off
    unsigned long long *item_stats;
    // optional work counters (diagnostics): [0] tile visits, [1] passes of
    // the lane-per-query path, [2] candidate (query, tile) pairs, [3] trips
    // of the lane-per-filter path, [4] items, [5] 4-filter groups tested by
    // the lane-per-query path, [6] its busy lanes summed over passes, [7]
    // its tile visits with at most 16 candidates; null when off
    unsigned long long *work;
};

// Marks the gather's padding records (no query).
constexpr uint32_t kPadQuery = 0xFFFFFFFFu;

// Shared memory of one matcher CTA (dynamic; ~54 KB, 4 CTAs per SM).
struct MatchSmem {
    // the item's query records; in two planes, so that the 16-byte reads of
    // scattered records spread over all banks (in 32-byte records each half
    // had every other 16 bytes to itself)
    uint4 q_lo[kItemQueries], q_hi[kItemQueries];
    HitRec rec[kMatchWarps][kWarpRecs];                  // staged hit records per warp
    // candidate lists per warp: 1024 / T bytes for each of the T tiles it
    // selects for at once, the chunks' candidates in chunk order (query index
    // in its chunk); trips read up to the next multiple of 4, what lies there
    // is any query of the item and its hits are dropped
    uint8_t list[kMatchWarps][kItemQueries];
    uint4 tf[kMatchWarps][kWords][kTile / 4];            // a warp's tile: word k of filters 4 g .. 4 g + 3
    uint64_t full, empty;
    uint32_t item;
    int fail;
    // thread 0's record of a copy in flight, with the parity of the phase
    // that completes it
    uint32_t inflight, inflight_par;
};

// 4 CTAs per SM: 228 KB of shared memory per SM, 1 KB of it reserved per CTA
static_assert(4 * (sizeof(MatchSmem) + 1024) <= 228 * 1024, "the matcher's shared memory must fit 4 CTAs per SM");

// Moves a warp's n staged records to the global record buffer (one atomic
// reserves their place; past the capacity they are only counted, and the
// host re-runs the batch with a larger buffer).  The records' key counts,
// the per-query key totals and the pair count are made here, with every lane
// at work, instead of at the few lanes that hit when a record is staged.
// Returns the lane's matching pairs.
__device__ __forceinline__ uint32_t flush_recs(HitRec *buf, uint32_t n, const MatchArgs &a, unsigned lane) {
    __syncwarp();
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(&a.counters[1], (unsigned long long)n);
    base = __shfl_sync(kFull, base, 0);
    const bool fits = base + n <= a.rec_cap;
    uint32_t pairs = 0;
    for (uint32_t i = lane; i < n; i += 32) {
        HitRec r = buf[i];
        r.nkeys = mask_keys(a.tile_keys[r.tile], r.mask, a.slot_key_off, r.tile);
        atomicAdd(&a.qkeys[r.query], r.nkeys);
        pairs += __popc(r.mask);
        if (fits) a.recs[base + i] = r;
    }
    __syncwarp();
    return pairs;
}

// A work item: up to kItemQueries consecutive queries of one partition's
// queue (its chunks' slices from zchunk on) against one segment of its tiles.
struct ItemRef {
    uint32_t qbase, nq, tb, te, zchunk;
};

__device__ __forceinline__ ItemRef locate(const MatchArgs &a, uint32_t item, uint32_t seg_tiles) {
    uint32_t lo = 0, hi = a.n_parts;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (a.item_off[mid] <= item) lo = mid;
        else hi = mid;
    }
    const uint32_t local = item - a.item_off[lo];
    if (a.part_order) lo = a.part_order[lo];
    ItemRef r;
    const uint32_t pq = a.part_count[lo];
    const uint32_t ngroups = (pq + kItemQueries - 1) / kItemQueries;
    const uint32_t group = local % ngroups, seg = local / ngroups;
    r.qbase = a.part_off[lo] + group * kItemQueries;
    r.nq = min((uint32_t)kItemQueries, pq - group * kItemQueries);
    r.tb = a.part_tile_begin[lo] + seg * seg_tiles;
    r.te = min(r.tb + seg_tiles, a.part_tile_begin[lo + 1]);
    r.zchunk = a.chunk_off[lo] + group * kItemChunks;
    return r;
}

// Thread 0: claim the next item and start the copies of its query records;
// the item id is published through the full barrier's phase completion.
// Returns whether copies are in flight.
__device__ __forceinline__ bool produce(const MatchArgs &a, uint32_t total, MatchSmem &S) {
    const uint32_t item = uint32_t(atomicAdd(&a.counters[0], 1ull));
    S.item = item;
    if (item < total) {
        const ItemRef r = locate(a, item, *a.seg);
        const uint32_t bytes = r.nq * sizeof(uint4);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_expect_tx(&S.full, 2 * bytes);
        tma_bulk_g2s(S.q_lo, a.queue_lo + r.qbase, bytes, &S.full);
        tma_bulk_g2s(S.q_hi, a.queue_hi + r.qbase, bytes, &S.full);
        return true;
    }
    mbar_arrive(&S.full);  // nothing to copy: complete the phase so consumers see the end
    return false;
}

// Lane per query: tests W candidates per lane (their words in q) against the
// tile's filters, 4 per step, and sets bit l of m[c] when candidate c holds
// filter l.  One broadcast 128-bit load gives word k of four filters; such a
// load takes two of the shared-memory pipe's cycles, so that with one
// candidate per lane the loads took as long as the LOP3s (48 against 56
// cycles per 128 tests and quarter SM).  A hit is added with a predicated
// add, which has a pipe of its own to go to; an or shares the LOP3s' (64
// against 53 cycles measured).
template <int W>
__device__ __forceinline__ void test_queries(const uint4 (*tf)[kTile / 4], uint32_t groups, const uint4 (&lo)[W],
                                             const uint4 (&hi)[W], uint32_t (&m)[W]) {
#pragma unroll
    for (int c = 0; c < W; ++c) m[c] = 0;
#pragma unroll
    for (int g = 0; g < kTile / 4; ++g) {
        if (g >= (int)groups) break;
        const uint4 w0 = tf[0][g], w1 = tf[1][g], w2 = tf[2][g], w3 = tf[3][g], w4 = tf[4][g], w5 = tf[5][g];
#pragma unroll
        for (int c = 0; c < W; ++c) {
            uint32_t x0 = w0.x & ~lo[c].x, x1 = w0.y & ~lo[c].x, x2 = w0.z & ~lo[c].x, x3 = w0.w & ~lo[c].x;
            x0 = andnot_or(w1.x, lo[c].y, x0);
            x1 = andnot_or(w1.y, lo[c].y, x1);
            x2 = andnot_or(w1.z, lo[c].y, x2);
            x3 = andnot_or(w1.w, lo[c].y, x3);
            x0 = andnot_or(w2.x, lo[c].z, x0);
            x1 = andnot_or(w2.y, lo[c].z, x1);
            x2 = andnot_or(w2.z, lo[c].z, x2);
            x3 = andnot_or(w2.w, lo[c].z, x3);
            x0 = andnot_or(w3.x, lo[c].w, x0);
            x1 = andnot_or(w3.y, lo[c].w, x1);
            x2 = andnot_or(w3.z, lo[c].w, x2);
            x3 = andnot_or(w3.w, lo[c].w, x3);
            x0 = andnot_or(w4.x, hi[c].x, x0);
            x1 = andnot_or(w4.y, hi[c].x, x1);
            x2 = andnot_or(w4.z, hi[c].x, x2);
            x3 = andnot_or(w4.w, hi[c].x, x3);
            x0 = andnot_or(w5.x, hi[c].y, x0);
            x1 = andnot_or(w5.y, hi[c].y, x1);
            x2 = andnot_or(w5.z, hi[c].y, x2);
            x3 = andnot_or(w5.w, hi[c].y, x3);
            add_if_zero(m[c], x0, 1u << (4 * g));
            add_if_zero(m[c], x1, 2u << (4 * g));
            add_if_zero(m[c], x2, 4u << (4 * g));
            add_if_zero(m[c], x3, 8u << (4 * g));
        }
    }
}

// The subset test.  Persistent CTAs take work items (partition, up to four
// consecutive 256-query chunks of its queue, segment of its tiles) from an
// atomic counter; thread 0 stages the item's query records with bulk TMA
// copies.  Each warp takes T tiles (<= 32 filters each) at a time, T x (the
// item's 32-query words, rounded up to a power of two) = 32 lanes: one tile
// for a full item, 32 tiles for an item of at most 32 queries, so that an
// item's selection is shared by as many tiles as its queries leave room for
// (one tile at a time took 32 visits where one is enough; one query against
// a million filters spent 33 us in the subset test):
//  * selection: the tile's 8 selector bits (bits every member holds); each
//    lane ORs the "lacks bit" slices of its tile and 32-query word, so a query
//    that lacks any of them is dropped; the remaining candidates go to the
//    tile's list (one byte per query, placed by a prefix sum over the tile's
//    words);
// then, tile by tile, over the candidates of all chunks together (one pass
// over the tile's filters for up to 1,024 queries: fuller passes and trips):
//  * many candidates, or an item of more than 512 queries: candidate queries
//    over the lanes (two per lane while more than 32 are left, then one), the tile's filters read from shared
//    memory (test_queries), the lane's hit mask over the tile built bit by
//    bit;
//  * few candidates: one filter per lane (the tile in registers), four
//    candidates per trip, one ballot per candidate for its hit mask;
//  * each (query, tile) with a hit becomes a 16-byte record (query, tile,
//    hit mask, key count), staged in a per-warp buffer and flushed with one
//    atomic; the flush counts the records' keys from the tiles' key-count bit
//    planes and adds them to qkeys[query] (for the prefix sum that places a
//    query's keys).
// The path per tile is chosen from the candidate count and the tile size
// (estimated instruction costs; the choice does not change results).
// COUNT: diagnostics instantiation that also tallies its work (a.work);
// TIMED: records each item's warp-cycles and hit records (a.item_stats).
template <bool COUNT, bool TIMED>
__global__ void __launch_bounds__(kMatchThreads, 4) k_match(MatchArgs a) {  // 4 CTAs per SM: up to 64 registers
    extern __shared__ __align__(128) unsigned char smem_raw[];
    MatchSmem &S = *reinterpret_cast<MatchSmem *>(smem_raw);
    const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t total = a.item_off[a.n_parts];
    if (tid == 0) {
        mbar_init(&S.full, 1);
        mbar_init(&S.empty, kMatchWarps);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        S.fail = 0;
        S.inflight = 0;
        S.inflight_par = 0;
    }
    __syncthreads();
    uint32_t w_tiles = 0, w_passes = 0, w_cand = 0, w_trips = 0, w_items = 0, w_groups = 0, w_lanes = 0, w_small = 0;
    uint32_t wn = 0;      // records staged by this warp (warp-uniform)
    uint32_t w_recs = 0;  // records this warp has produced (warp-uniform)
    uint32_t pairs = 0;   // matching (query, filter) pairs counted by this lane
    const uint32_t lane_lt = (1u << lane) - 1u;
    uint32_t *tfw = reinterpret_cast<uint32_t *>(S.tf[warp]);
    uint8_t *list = S.list[warp];
    HitRec *rec = S.rec[warp];
    // stages one record for every lane with a hit mask m
    auto stage = [&](uint32_t m, uint32_t query, uint32_t t) {
        const uint32_t wm = __ballot_sync(kFull, m != 0);
        if (wm == 0) return;
        const uint32_t k = __popc(wm);
        if (wn + k > (uint32_t)kWarpRecs) {
            pairs += flush_recs(rec, wn, a, lane);
            wn = 0;
        }
        if (m) rec[wn + __popc(wm & lane_lt)] = HitRec{query, t, m, 0u};
        wn += k;
        if (TIMED) w_recs += k;
    };
    for (uint32_t it = 0;; ++it) {
        // stage the next item once every warp has released the buffers
        // (they held item it - 1); thread 0 keeps track of the copies in
        // flight, so that none still targets this CTA's shared memory when
        // it exits
        if (tid == 0) {
            bool ok = true;
            if (it >= 1) ok = mbar_wait(&S.empty, (it - 1) & 1);
            if (ok) {
                S.inflight = produce(a, total, S) ? 1u : 0u;
                S.inflight_par = it & 1;
            } else {
                atomicOr(&a.counters[2], 1ull);
                S.fail = 1;
            }
        }
        // every exit is taken by whole warps (record flushes use the full warp)
        const bool got = mbar_wait(&S.full, it & 1);
        if (tid == 0 && got) S.inflight = 0;
        if (!__all_sync(kFull, got)) {
            if (lane == 0) atomicOr(&a.counters[2], 2ull);
            break;
        }
        const uint32_t item = S.item;
        if (__any_sync(kFull, item >= total || S.fail)) break;
        const ItemRef r = locate(a, item, *a.seg);
        if (COUNT) ++w_items;
        long long item_c0 = 0;
        uint32_t item_recs0 = 0;
        if (TIMED) {
            item_c0 = clock64();
            item_recs0 = w_recs;
        }
        // lanes per tile: the item's 32-query words, as a power of two
        // (all lanes for more than 512 queries).  Wide items are compiled by
        // themselves: with the lanes' roles known, the scan unrolled, no loop
        // over tiles and only the lane-per-query path (few of their tiles
        // have few candidates), 65,536 queries on ten million filters take
        // 24.9 ms instead of 27.1.  More cases, or the second path, cost more
        // in the instruction cache than they save: 500 queries, whose items
        // have 4 to 16 words, went from 0.58 to 0.86 ms with a case for 16.
        const uint32_t words = (r.nq + 31) >> 5;
        auto all_tiles = [&](auto wide) {
            constexpr bool kWide = decltype(wide)::value;
            const uint32_t lg = kWide ? 5u : words > 1 ? 32 - __clz(words - 1) : 0u, tiles = 32u >> lg;
            const uint32_t wi = lane & ((1u << lg) - 1u), gi = lane >> lg;  // the lane's word, its tile of the step
            const uint32_t last = lane | ((1u << lg) - 1u);                   // the last lane of its tile
            // queries of the lane's word, and its slices
            const uint32_t live = wi * 32 + 32 <= r.nq ? kFull : wi * 32 >= r.nq ? 0u : (1u << (r.nq - wi * 32)) - 1u;
            const uint32_t *zl = a.slices + (size_t(r.zchunk) + (wi >> 3)) * kSliceWords + (wi & 7);
            for (uint32_t t0 = r.tb + warp * tiles; t0 < r.te; t0 += kMatchWarps * tiles) {
                const uint32_t tq = t0 + gi;
                uint32_t cand = 0, tcount = 0;
                if (kWide || tq < r.te) {
                    const TileInfo ti = a.tile_info[tq];
                    tcount = ti.count;
                    if (live) {  // words past the item's queries have no slices
                        const uint32_t lack =
                            __ldg(&zl[(ti.sel[0] & 0xFFu) * 8]) | __ldg(&zl[((ti.sel[0] >> 8) & 0xFFu) * 8]) |
                            __ldg(&zl[((ti.sel[0] >> 16) & 0xFFu) * 8]) | __ldg(&zl[(ti.sel[0] >> 24) * 8]) |
                            __ldg(&zl[(ti.sel[1] & 0xFFu) * 8]) | __ldg(&zl[((ti.sel[1] >> 8) & 0xFFu) * 8]) |
                            __ldg(&zl[((ti.sel[1] >> 16) & 0xFFu) * 8]) | __ldg(&zl[(ti.sel[1] >> 24) * 8]);
                        cand = ~lack & live;
                    }
                }
                if (COUNT) w_tiles += __popc(__ballot_sync(kFull, tq < r.te && wi == 0));  // lane 0 reports
                // candidate lists (query index in its chunk, one byte each): a
                // prefix sum over each tile's words places every lane's queries,
                // from the word's highest down
                const uint32_t cnt = __popc(cand);
                uint32_t incl = cnt;
#pragma unroll
                for (uint32_t o = 1; o < 32; o <<= 1) {
                    if (!kWide && o >= (1u << lg)) break;
                    const uint32_t v = __shfl_up_sync(kFull, incl, o);
                    if (wi >= o) incl += v;
                }
                {
                    uint8_t *at = list + ((gi << lg) << 5) + incl;
                    while (cand) {
                        const uint32_t bit = 31u - __clz(cand);
                        cand ^= 1u << bit;
                        *--at = uint8_t(wi * 32 + bit);
                    }
                }
                __syncwarp();
                uint32_t todo = kWide ? 1u << 31 : __ballot_sync(kFull, lane == last && incl != 0);
                for (; todo; todo = kWide ? 0u : todo & (todo - 1)) {
                    const uint32_t end = kWide ? 31u : __ffs(todo) - 1, first = end & ~((1u << lg) - 1u);  // the tile's lanes
                    const uint32_t n = __shfl_sync(kFull, incl, end), count = kWide ? tcount : __shfl_sync(kFull, tcount, first);
                    if (kWide && n == 0) break;
                    const uint32_t t = t0 + (end >> lg);
                    // list positions where chunks 1 .. kItemChunks - 1 begin: the
                    // candidate at position x is in chunk sum_c (x >= cb[c])
                    uint32_t cb[kItemChunks - 1];
#pragma unroll
                    for (int c = 0; c + 1 < kItemChunks; ++c) cb[c] = __shfl_sync(kFull, incl, min(first + 8 * c + 7, end));
                    auto query_at = [&](uint32_t x, uint32_t in_chunk) {
                        uint32_t c = 0;
#pragma unroll
                        for (int k = 0; k + 1 < kItemChunks; ++k) c += x >= cb[k] ? (uint32_t)kChunk : 0u;
                        return c + in_chunk;
                    };
                    if (COUNT) w_cand += n;  // the warp's candidates (lane 0 reports)
                    const uint8_t *lst = list + (first << 5);
                    uint32_t f[kWords];
#pragma unroll
                    for (int k = 0; k < kWords; ++k) f[k] = __ldg(&a.tile_words[(size_t(t) * kWords + k) * kTile + lane]);
                    const uint32_t vm = count >= 32u ? kFull : (1u << count) - 1u;  // lanes holding a filter
                    const uint32_t groups = (count + 3) >> 2;
                    const bool per_query = kWide || ((n + 31) >> 5) * (16u + 40u * groups) < ((n + 3) >> 2) * a.fpl_trip_cost;
                    if (per_query) {
#pragma unroll
                        for (int k = 0; k < kWords; ++k) tfw[k * kTile + lane] = f[k];
                        __syncwarp();
                        uint32_t p0 = 0;
                        for (; p0 + 32 < n; p0 += 64) {
                            const uint32_t j0 = p0 + lane, j1 = j0 + 32;
                            const uint32_t i0 = query_at(j0, lst[j0]), i1 = j1 < n ? query_at(j1, lst[j1]) : 0u;
                            const uint4 lo[2] = {S.q_lo[i0], S.q_lo[i1]}, hi[2] = {S.q_hi[i0], S.q_hi[i1]};
                            uint32_t m[2];
                            test_queries<2>(S.tf[warp], groups, lo, hi, m);
                            if (COUNT) {
                                w_passes += 2;
                                w_groups += 2 * groups;
                                w_lanes += min(64u, n - p0);
                            }
                            stage(m[0] & vm, hi[0].z, t);
                            stage(j1 < n ? m[1] & vm : 0u, hi[1].z, t);
                        }
                        if (p0 < n) {
                            const uint32_t j0 = p0 + lane, i0 = j0 < n ? query_at(j0, lst[j0]) : 0u;
                            const uint4 lo[1] = {S.q_lo[i0]}, hi[1] = {S.q_hi[i0]};
                            uint32_t m[1];
                            test_queries<1>(S.tf[warp], groups, lo, hi, m);
                            if (COUNT) {
                                ++w_passes;
                                w_groups += groups;
                                w_lanes += n - p0;
                                if (p0 == 0 && n <= 16) ++w_small;
                            }
                            stage(j0 < n ? m[0] & vm : 0u, hi[0].z, t);
                        }
                    } else {
                        const bool lane_valid = lane < count;
                        for (uint32_t j = 0; j < n; j += 4) {
                            if (COUNT) ++w_trips;
                            const uint32_t idx4 = *reinterpret_cast<const uint32_t *>(lst + j);
                            const uint32_t ia = query_at(j, idx4 & 0xFFu), ib = query_at(j + 1, (idx4 >> 8) & 0xFFu);
                            const uint32_t ic = query_at(j + 2, (idx4 >> 16) & 0xFFu), id = query_at(j + 3, idx4 >> 24);
                            const uint4 p0 = S.q_lo[ia], p1 = S.q_hi[ia];
                            const uint4 q0 = S.q_lo[ib], q1 = S.q_hi[ib];
                            const uint4 r0 = S.q_lo[ic], r1 = S.q_hi[ic];
                            const uint4 u0 = S.q_lo[id], u1 = S.q_hi[id];
                            uint32_t x0 = f[0] & ~p0.x, x1 = f[0] & ~q0.x, x2 = f[0] & ~r0.x, x3 = f[0] & ~u0.x;
                            x0 = andnot_or(f[1], p0.y, x0);
                            x1 = andnot_or(f[1], q0.y, x1);
                            x2 = andnot_or(f[1], r0.y, x2);
                            x3 = andnot_or(f[1], u0.y, x3);
                            x0 = andnot_or(f[2], p0.z, x0);
                            x1 = andnot_or(f[2], q0.z, x1);
                            x2 = andnot_or(f[2], r0.z, x2);
                            x3 = andnot_or(f[2], u0.z, x3);
                            x0 = andnot_or(f[3], p0.w, x0);
                            x1 = andnot_or(f[3], q0.w, x1);
                            x2 = andnot_or(f[3], r0.w, x2);
                            x3 = andnot_or(f[3], u0.w, x3);
                            x0 = andnot_or(f[4], p1.x, x0);
                            x1 = andnot_or(f[4], q1.x, x1);
                            x2 = andnot_or(f[4], r1.x, x2);
                            x3 = andnot_or(f[4], u1.x, x3);
                            x0 = andnot_or(f[5], p1.y, x0);
                            x1 = andnot_or(f[5], q1.y, x1);
                            x2 = andnot_or(f[5], r1.y, x2);
                            x3 = andnot_or(f[5], u1.y, x3);
                            // common case: no hit among the four (one min chain, one vote)
                            if (!__any_sync(kFull, lane_valid && min(min(x0, x1), min(x2, x3)) == 0)) continue;
                            // warp-uniform from here: one ballot per candidate gives the
                            // tile's hit mask for that query; lane k < 4 stages record k
                            // (what lies past the list is dropped)
                            const uint32_t b0 = __ballot_sync(kFull, x0 == 0) & vm;
                            const uint32_t b1 = __ballot_sync(kFull, x1 == 0) & vm;
                            const uint32_t b2 = __ballot_sync(kFull, x2 == 0) & vm;
                            const uint32_t b3 = __ballot_sync(kFull, x3 == 0) & vm;
                            const uint32_t mine = lane == 0 ? b0 : lane == 1 ? b1 : lane == 2 ? b2 : b3;
                            const uint32_t qid = lane == 0 ? p1.z : lane == 1 ? q1.z : lane == 2 ? r1.z : u1.z;
                            stage(lane < 4 && j + lane < n ? mine : 0u, qid, t);
                        }
                    }
                    __syncwarp();  // the tile buffer is rebuilt for the next tile
                }
                __syncwarp();  // the lists are rebuilt for the next tiles
            }
        };
        if (words > 16) all_tiles(std::true_type{});
        else all_tiles(std::false_type{});
        __syncwarp();
        if (TIMED && lane == 0) {
            atomicAdd(&a.item_stats[2 * size_t(item)], (unsigned long long)(clock64() - item_c0));
            atomicAdd(&a.item_stats[2 * size_t(item) + 1], (unsigned long long)(w_recs - item_recs0));
        }
        if (lane == 0) mbar_arrive(&S.empty);
    }
    if (wn) pairs += flush_recs(rec, wn, a, lane);
    pairs = __reduce_add_sync(kFull, pairs);
    if (lane == 0 && pairs) atomicAdd(&a.counters[3], (unsigned long long)pairs);
    if (COUNT && lane == 0) {
        atomicAdd(&a.work[0], (unsigned long long)w_tiles);
        atomicAdd(&a.work[1], (unsigned long long)w_passes);
        atomicAdd(&a.work[2], (unsigned long long)w_cand);
        atomicAdd(&a.work[3], (unsigned long long)w_trips);
        atomicAdd(&a.work[5], (unsigned long long)w_groups);
        atomicAdd(&a.work[6], (unsigned long long)w_lanes);
        atomicAdd(&a.work[7], (unsigned long long)w_small);
        if (warp == 0) atomicAdd(&a.work[4], (unsigned long long)w_items);
    }
    // no copy may still target this CTA's shared memory when it exits: after
    // a failed wait, wait (bounded) for the copies still in flight
    if (tid == 0 && S.inflight && !mbar_wait(&S.full, S.inflight_par)) atomicOr(&a.counters[2], 4ull);
}

// Launches the subset test on grid CTAs (its shared memory is above the
// 48 KB static limit, so the size is set on the kernel first).
template <bool COUNT, bool TIMED>
inline void launch_match_t(const MatchArgs &a, unsigned grid, cudaStream_t st) {
    TM_CUDA(cudaFuncSetAttribute(k_match<COUNT, TIMED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(sizeof(MatchSmem))));
    TM_CUDA(cudaFuncSetAttribute(k_match<COUNT, TIMED>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 int(cudaSharedmemCarveoutMaxShared)));
    k_match<COUNT, TIMED><<<grid, kMatchThreads, sizeof(MatchSmem), st>>>(a);
}

template <bool COUNT>
inline void launch_match(const MatchArgs &a, unsigned grid, cudaStream_t st) {
    if (a.item_stats) launch_match_t<COUNT, true>(a, grid, st);
    else launch_match_t<COUNT, false>(a, grid, st);
}

// ---------------------------------------------------------------------------
// Key gather
// ---------------------------------------------------------------------------
constexpr int kFillPerLane = 2;  // records per lane and warp step (loads in flight)
constexpr int kFillCtas = 6;     // resident per SM, at least (register budget)

constexpr int kFillThreads = 256;
constexpr int kFillWarps = kFillThreads / 32;
constexpr int kFillStep = 32 * kFillPerLane;  // records per warp step
// The block variant of the gather: most records per block, and the most queries
// of a batch that takes it (4 bytes of shared memory each).
constexpr uint32_t kFillBlockRecs = 2048;
constexpr uint32_t kFillBlockQueries = 2048;
// Keys per record from which the gather is the one that looks for long runs,
// and keys of a batch of 32 runs from which it copies them one by one.
constexpr uint32_t kLongRecord = 32;
constexpr uint32_t kLongBatch = 32 * 128;

// Owners of 32 consecutive positions p0 + lane, when lane i owns a non-empty
// stretch that begins at `start` (increasing with i; live: the lane has one):
// the begins inside the window as a bit mask, and the lanes that began before
// it.  Eight instructions, where a binary search by shuffles takes five
// rounds of three on the shared-memory pipe.
__device__ __forceinline__ uint32_t owner_of(uint32_t start, bool live, uint32_t p0, uint32_t lane_le) {
    const uint32_t begins = __reduce_or_sync(kFull, live && start >= p0 && start - p0 < 32u ? 1u << (start - p0) : 0u);
    const uint32_t before = __popc(__ballot_sync(kFull, live && start < p0));
    return before + __popc(begins & lane_le) - 1u;
}

// Copies every record's keys into its query's range (qoff).  Each record's
// keys are reserved on the query's cursor (qcursor, zeroed by the caller).
// The table keeps keys in slot order, so each run of adjacent hit bits
// [lo, hi) of a record's mask is the key range [o[lo], o[hi]) of the tile's
// slot offsets o.  A warp takes 32 x kFillPerLane records per step and
// numbers all their runs (a prefix sum over the lanes' run counts); lane i of
// a batch then takes run 32 b + i: the lane whose records hold it (owner_of),
// the record from shared memory, the run's first bit, its key range from the
// slot offsets, and its place in the record's output from the keys of the hit
// bits below it (the tile's key-count planes).  The warp copies the batch's
// runs together, 32 keys per step (a prefix sum over the run lengths and, for
// key j, the run that owns it), so the stores coalesce and a record with
// several runs costs no extra pass over the warp.
//
// BLOCK: a CTA takes block_recs consecutive records, sums their keys per
// query in shared memory and reserves each query's keys with one global
// atomic.  Atomics on one address follow one another, and in a batch of few
// queries the heaviest holds a good part of all records: 500 queries of the
// ten-million table (1.8 M records) took 272 us, six times the time per
// record of a batch of 20,011.
//
// LONG: batches of 32 runs of kLongBatch keys or more are copied run by run,
// four loads in flight, where 32 keys of all runs at a time wait for each load.
// 20,000 queries with one run each, us: runs of 100 keys 137 as short ones and
// 142 as long ones, of 150 159 and 125, of 400 256 and 150, of 2,000 927 and
// 323.  An instantiation of its own for tables with that many keys per record:
// the code beside the short way costs batches of short runs 0.3 to 0.6% of
// their whole time.
template <bool BLOCK, bool LONG>
__global__ void __launch_bounds__(kFillThreads, kFillCtas) k_key_fill(
    const HitRec *__restrict__ recs, const unsigned long long *__restrict__ counters,
    const uint32_t *__restrict__ slot_key_off, const TileKeys *__restrict__ tile_keys, const uint32_t *__restrict__ tkeys,
    const uint64_t *__restrict__ qoff, uint32_t *__restrict__ qcursor, uint32_t nq, uint32_t block_recs,
    uint32_t *__restrict__ out) {
    extern __shared__ uint32_t s_cur[];  // BLOCK: [nq] the block's cursor per query
    // per warp and record of the step: tile, hit mask, keys, runs of the
    // lane's earlier records; and the record's first output position
    __shared__ uint4 s_rec[kFillWarps][kFillStep];
    __shared__ unsigned long long s_dst[kFillWarps][kFillStep];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t lane_le = (2u << lane) - 1u;
    const unsigned long long n = counters[1];
    // records [base, end) by the calling warp, kFillStep at most
    auto step = [&](unsigned long long base, unsigned long long end) {
        HitRec r[kFillPerLane];
#pragma unroll
        for (int j = 0; j < kFillPerLane; ++j) {
            const unsigned long long i = base + j * 32 + lane;
            r[j] = i < end ? recs[i] : HitRec{kPadQuery, 0u, 0u, 0u};
        }
        uint32_t nruns = 0;
        unsigned long long dst[kFillPerLane];
#pragma unroll
        for (int j = 0; j < kFillPerLane; ++j) {
            const bool live = r[j].query != kPadQuery;
            const uint32_t m = live ? r[j].mask : 0u;
            dst[j] = live ? qoff[r[j].query] + atomicAdd(BLOCK ? &s_cur[r[j].query] : &qcursor[r[j].query], r[j].nkeys) : 0ull;
            s_rec[warp][j * 32 + lane] = make_uint4(r[j].tile, m, r[j].nkeys, nruns);
            nruns += __popc(m & ~(m << 1));  // run starts
        }
        const uint32_t incl = warp_incl_scan(nruns);
        const uint32_t total = __shfl_sync(kFull, incl, 31);
        const uint32_t excl = incl - nruns;
        __syncwarp();
        for (uint32_t rb = 0; rb < total; rb += 32) {
            const uint32_t ri = rb + lane;
            const uint32_t owner = owner_of(excl, nruns != 0, rb, lane_le);
            const uint32_t oexcl = __shfl_sync(kFull, excl, owner);
            const bool have = ri < total;
            uint32_t slot = owner, src = 0, end_key = 0, below = 0, t = 0, nk = 0;
            bool last = true;
            TileKeys tk{{0u, 0u, 0u}, 0u};
            if (have) {
                const uint32_t k = ri - oexcl;  // run number within the owner lane's records
                // its record: the last whose earlier-run count is <= k
#pragma unroll
                for (int jj = 1; jj < kFillPerLane; ++jj)
                    if (s_rec[warp][jj * 32 + owner].w <= k) slot = jj * 32 + owner;
                const uint4 rc = s_rec[warp][slot];
                const uint32_t m = rc.y;
                t = rc.x;
                nk = rc.z;
                uint32_t starts = m & ~(m << 1);
                for (uint32_t i = k - rc.w; i; --i) starts &= starts - 1;  // few: most records have one run
                const uint32_t lo = __ffs(starts) - 1u;
                const uint32_t above = ~(m >> lo);  // first clear bit from lo on (none: the run ends the tile)
                const uint32_t hi = above ? lo + __ffs(above) - 1u : 32u;
                const uint32_t *o = slot_key_off + size_t(t) * kTile;
                below = m & ((1u << lo) - 1u);  // hit bits of the earlier runs
                last = hi >= 32u || (m >> hi) == 0u;
                src = o[lo];
                if (!last) end_key = o[hi];
                if (below) tk = tile_keys[t];
            }
            if (rb == 0) {
                // the cursor atomics' results, published once the first
                // batch's offset loads are in flight
#pragma unroll
                for (int j = 0; j < kFillPerLane; ++j) s_dst[warp][j * 32 + lane] = dst[j];
                __syncwarp();
            }
            uint32_t len = 0;
            unsigned long long d = 0;
            if (have) {
                const uint32_t bk = below ? mask_keys(tk, below, slot_key_off, t) : 0u;
                len = last ? nk - bk : end_key - src;
                d = s_dst[warp][slot] + bk;
            }
            // the batch's runs, copied together: key j of the batch comes from
            // src - start + j and goes to d - start + j of its run
            const uint32_t kin = warp_incl_scan(len);
            const uint32_t keys = __shfl_sync(kFull, kin, 31);
            const uint32_t start = kin - len;
            if (LONG && keys >= kLongBatch) {
                for (uint32_t runs = __ballot_sync(kFull, len != 0); runs; runs &= runs - 1) {
                    const uint32_t ro = __ffs(runs) - 1;
                    const uint32_t n_run = __shfl_sync(kFull, len, ro);
                    const uint32_t *from = tkeys + __shfl_sync(kFull, src, ro);
                    uint32_t *to = out + __shfl_sync(kFull, d, ro);
                    uint32_t k = lane;
                    for (; k + 96 < n_run; k += 128) {
                        const uint32_t v0 = from[k], v1 = from[k + 32], v2 = from[k + 64], v3 = from[k + 96];
                        to[k] = v0;
                        to[k + 32] = v1;
                        to[k + 64] = v2;
                        to[k + 96] = v3;
                    }
                    for (; k < n_run; k += 32) to[k] = from[k];
                }
                continue;
            }
            src -= start;
            d -= start;
            for (uint32_t j0 = 0; j0 < keys; j0 += 32) {
                const uint32_t kk = j0 + lane;
                const uint32_t ro = owner_of(start, len != 0, j0, lane_le);
                const uint32_t osrc = __shfl_sync(kFull, src, ro);
                const unsigned long long odst = __shfl_sync(kFull, d, ro);
                if (kk < keys) out[odst + kk] = tkeys[osrc + kk];
            }
        }
        __syncwarp();  // the shared entries are rewritten by the next step
    };
    if constexpr (BLOCK) {
        for (unsigned long long b0 = (unsigned long long)blockIdx.x * block_recs; b0 < n;
             b0 += (unsigned long long)gridDim.x * block_recs) {
            const unsigned long long b1 = min(n, b0 + block_recs);
            for (uint32_t q = threadIdx.x; q < nq; q += kFillThreads) s_cur[q] = 0;
            __syncthreads();
            for (unsigned long long i = b0 + threadIdx.x; i < b1; i += kFillThreads) {
                const HitRec r = recs[i];
                atomicAdd(&s_cur[r.query], r.nkeys);
            }
            __syncthreads();
            for (uint32_t q = threadIdx.x; q < nq; q += kFillThreads) {
                const uint32_t c = s_cur[q];
                if (c) s_cur[q] = atomicAdd(&qcursor[q], c);
            }
            __syncthreads();
            for (unsigned long long base = b0 + warp * kFillStep; base < b1; base += kFillWarps * kFillStep) step(base, b1);
            __syncthreads();  // the cursors are rewritten for the next block
        }
    } else {
        const unsigned long long warps = (unsigned long long)gridDim.x * kFillWarps;
        for (unsigned long long base = ((unsigned long long)blockIdx.x * kFillWarps + warp) * kFillStep; base < n;
             base += warps * kFillStep)
            step(base, n);
    }
}

// Gathers the `keys` keys of n_recs records of nq queries (qcursor zeroed).
inline void launch_key_fill(const DevTable &t, const HitRec *recs, const unsigned long long *counters,
                            unsigned long long n_recs, uint64_t keys, const uint64_t *qoff, uint32_t *qcursor, uint32_t nq,
                            uint32_t *out, int sm_count, cudaStream_t st) {
    const unsigned most = unsigned(sm_count) * 16;
    const bool longer = keys >= kLongRecord * n_recs;
    if (nq <= kFillBlockQueries) {
        // few records are spread over the SMs, a warp's step of them each at
        // least: they may have thousands of keys each (2,048 queries with a run
        // of 400 keys each: 688 us in one block of 2,048 records, 116 so)
        const unsigned long long per_sm = (n_recs + sm_count - 1) / sm_count;
        const uint32_t block_recs = std::min(kFillBlockRecs, blocks_for(std::max(per_sm, 1ull), kFillStep) * kFillStep);
        const unsigned grid = std::max(1u, std::min(blocks_for(n_recs, block_recs), most));
        (longer ? k_key_fill<true, true> : k_key_fill<true, false>)<<<grid, kFillThreads, nq * sizeof(uint32_t), st>>>(
            recs, counters, t.slot_key_off.p, t.tile_keys.p, t.keys.p, qoff, qcursor, nq, block_recs, out);
    } else {
        const unsigned grid = std::max(1u, std::min(blocks_for(n_recs, kFillThreads * kFillPerLane), most));
        (longer ? k_key_fill<false, true> : k_key_fill<false, false>)<<<grid, kFillThreads, 0, st>>>(
            recs, counters, t.slot_key_off.p, t.tile_keys.p, t.keys.p, qoff, qcursor, nq, 0, out);
    }
    TM_CHECK_LAUNCH();
}

// ---------------------------------------------------------------------------
// match_unique
// ---------------------------------------------------------------------------
// Two routes.  Keys of a small space [0, 32 * words) are marked in a bitmap
// per query, which is then read out in order; others, and few keys in a space
// that is not so small, are sorted.
constexpr uint32_t kBitmapMaxWords = 12288;  // 48 KB of shared memory

// Words between two queries' bitmaps (16-byte rows).
__host__ __device__ inline uint32_t bitmap_stride(uint32_t words) { return (words + 3u) & ~3u; }

// Marks a query's keys in a bitmap (built in shared memory, one CTA per
// query), stores it and counts its bits.  Keeping the bitmap (8 KB per query
// for 16-bit keys) lets the read-out write to the result's own place once
// the counts are known, where writing keys per query and moving them
// together afterwards took 428 us for 20,011 queries of 2,580 keys (mark,
// read-out and move), and the two kernels here take 98 + 163 us: reading
// the keys, the bitmaps' way out and back and the result are about 0.7 GB.
// A block's time is the latency of its few steps, so a batch of many
// queries wants small blocks, eight to an SM (256 threads: 98 us against 153
// with 512 and 209 with 1,024); where all queries are resident at once, the
// longest result is the kernel's time and wants many threads (500 queries
// of the ten-million table: 89, 53 and 37 us).
__global__ void __launch_bounds__(1024) k_unique_mark(const uint32_t *__restrict__ keys,
                                                              const uint64_t *__restrict__ qoff, uint32_t words,
                                                              uint32_t *__restrict__ bitmaps, uint32_t *__restrict__ ucount) {
    extern __shared__ uint4 bm4[];
    __shared__ uint32_t s_count;
    uint32_t *bm = reinterpret_cast<uint32_t *>(bm4);
    const uint32_t q = blockIdx.x;
    const uint64_t b = qoff[q], e = qoff[q + 1];
    if (e == b) {  // no bits, and no read-out
        if (threadIdx.x == 0) ucount[q] = 0;
        return;
    }
    const uint32_t rows = bitmap_stride(words) >> 2;
    for (uint32_t i = threadIdx.x; i < rows; i += blockDim.x) bm4[i] = make_uint4(0, 0, 0, 0);
    if (threadIdx.x == 0) s_count = 0;
    __syncthreads();
    auto mark = [&](uint32_t k) { atomicOr(&bm[k >> 5], 1u << (k & 31)); };
    auto mark4 = [&](const uint4 &v) {
        mark(v.x);
        mark(v.y);
        mark(v.z);
        mark(v.w);
    };
    // whole groups of four keys by 16-byte loads, two in flight per thread;
    // the ragged ends one key at a time
    const uint64_t b4 = min(e, (b + 3) & ~uint64_t(3)), e4 = max(b4, e & ~uint64_t(3));
    if (b + threadIdx.x < b4) mark(keys[b + threadIdx.x]);
    if (e4 + threadIdx.x < e) mark(keys[e4 + threadIdx.x]);
    const uint4 *k4 = reinterpret_cast<const uint4 *>(keys);
    uint64_t i = (b4 >> 2) + threadIdx.x;
    for (; i + blockDim.x < (e4 >> 2); i += 2 * blockDim.x) {
        const uint4 v0 = k4[i], v1 = k4[i + blockDim.x];
        mark4(v0);
        mark4(v1);
    }
    if (i < (e4 >> 2)) mark4(k4[i]);
    __syncthreads();
    uint4 *out = reinterpret_cast<uint4 *>(bitmaps + size_t(q) * (rows * 4));
    uint32_t c = 0;
    for (uint32_t r = threadIdx.x; r < rows; r += blockDim.x) {
        const uint4 v = bm4[r];
        out[r] = v;
        c += __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
    }
    c = __reduce_add_sync(kFull, c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(&s_count, c);
    __syncthreads();
    if (threadIdx.x == 0) ucount[q] = s_count;
}

// Reads a query's bitmap out in order into its place of the result (one CTA
// per query, of as many warps as the bitmap has rounds, eight at most).  Warp w
// takes words [w * per, (w + 1) * per), 64 at a time,
// two per lane: a prefix sum over the lanes' popcounts places each lane's
// keys in a per-warp buffer (11-bit positions in the round's 2,048), which
// the warp then writes out 32 consecutive keys per store.
template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32) k_unique_expand(const uint32_t *__restrict__ bitmaps,
                                                                  const uint64_t *__restrict__ uoff, uint32_t words,
                                                                  uint32_t *__restrict__ out) {
    __shared__ uint16_t s_stage[WARPS][2048];
    __shared__ uint32_t s_sum[WARPS];
    const uint32_t q = blockIdx.x;
    const uint64_t o = uoff[q];
    if (uoff[q + 1] == o) return;
    // rows of two words; the stride is even and its padding words are zero
    const uint32_t rows = bitmap_stride(words) >> 1;
    const uint2 *bm = reinterpret_cast<const uint2 *>(bitmaps) + size_t(q) * rows;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t per = ((rows + WARPS - 1) / WARPS + 31) & ~31u;
    const uint32_t r0 = min(rows, warp * per), r1 = min(rows, r0 + per);
    uint32_t c = 0;
    for (uint32_t r = r0 + lane; r < r1; r += 32) {
        const uint2 v = bm[r];
        c += __popc(v.x) + __popc(v.y);
    }
    c = __reduce_add_sync(kFull, c);
    if (lane == 0) s_sum[warp] = c;
    __syncthreads();
    uint32_t *d = out + o;
#pragma unroll
    for (int k = 0; k < WARPS; ++k)
        if (k < int(warp)) d += s_sum[k];
    uint16_t *stage = s_stage[warp];
    for (uint32_t r = r0; r < r1; r += 32) {
        const uint2 v = r + lane < r1 ? bm[r + lane] : make_uint2(0u, 0u);
        const uint32_t cnt = __popc(v.x) + __popc(v.y);
        const uint32_t incl = warp_incl_scan(cnt);
        const uint32_t total = __shfl_sync(kFull, incl, 31);
        // from the highest key down: one find per key (two words per lane
        // even out the lanes' counts: 163 us against 187 with one)
        uint16_t *at = stage + incl, *end = at - cnt;
        uint32_t x = v.y, next = v.x, base = lane * 64 + 32;
        while (at != end) {
            if (x == 0) {
                x = next;
                base -= 32;
            }
            const uint32_t bit = 31u - __clz(x);
            x ^= 1u << bit;
            *--at = uint16_t(base + bit);
        }
        __syncwarp();
        for (uint32_t j = lane; j < total; j += 32) d[j] = r * 64 + stage[j];
        __syncwarp();  // the buffer is rewritten by the next round
        d += total;
    }
}

// The sorting route: a stable LSD radix sort of each query's keys, 8 bits
// per pass, one CTA per query; then the first of each run of equal keys goes
// to ukeys[b ..).  Queries of up to SMEM_KEYS keys ping-pong between two
// buffers in shared memory, longer ones between keys and ukeys.  Warp w
// holds the w-th stretch of the keys, so ranks come from per-warp digit
// counts (a prefix sum over digits, then warps) and, within 32 keys, from
// the lanes that hold the same digit.  Most results are short, and a small
// block per query keeps many of them resident; the queries above
// kSortSmallKeys keys are on a list, and a kernel of their own gives them 1,024
// threads each.  Both are bound by the shared-memory steps of the ranking:
// 2,000 queries of 1,070 32-bit keys take 82 + 83 us (the few long results),
// where one thread per stretch with 4-bit digits in global memory took 650.
constexpr int kSortSmallThreads = 256, kSortLargeThreads = 1024;
constexpr uint32_t kSortSmallKeys = 4096, kSortLargeKeys = 22528;
template <int THREADS, uint32_t SMEM_KEYS>
constexpr int kSortSmem = int(sizeof(uint32_t)) * (THREADS / 32 * 256 + 2 * int(SMEM_KEYS));

template <int THREADS, uint32_t SMEM_KEYS>
__device__ __forceinline__ void sort_query(uint32_t *keys, uint64_t b, uint32_t n, uint32_t *ukeys, uint32_t *ucount,
                                           int key_bits) {
    constexpr int kWarps = THREADS / 32;
    extern __shared__ uint32_t s_dyn[];
    uint32_t *s_cnt = s_dyn;                 // [kWarps][256] digit counts, then output positions
    uint32_t *s_key = s_dyn + kWarps * 256;  // [2][SMEM_KEYS]
    __shared__ uint32_t s_part[kWarps];
    const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool local = n <= SMEM_KEYS;
    uint32_t *src = keys + b, *dst = ukeys + b;
    if (local) {
        for (uint32_t i = tid; i < n; i += THREADS) s_key[i] = src[i];
        src = s_key;
        dst = s_key + SMEM_KEYS;
    }
    // the warp's stretch: whole groups of 32 keys
    const uint32_t per = ((n + kWarps - 1) / kWarps + 31) & ~31u;
    const uint32_t r0 = min(uint64_t(n), uint64_t(warp) * per), r1 = min(uint64_t(n), uint64_t(r0) + per);
    uint32_t *cnt = s_cnt + warp * 256;
    for (int shift = 0; shift < key_bits; shift += 8) {
        for (int i = lane; i < 256; i += 32) cnt[i] = 0;
        __syncthreads();  // also: the keys are in place
        for (uint32_t i = r0 + lane; i < r1; i += 32) atomicAdd(&cnt[(src[i] >> shift) & 255u], 1u);
        __syncthreads();
        // positions: thread t holds digit t (256 threads); a digit that
        // holds every key leaves the order as it is
        uint32_t tot = 0;
        if (tid < 256) {
            for (int w = 0; w < kWarps; ++w) tot += s_cnt[w * 256 + tid];
        }
        if (__syncthreads_or(tid < 256 && tot == n)) continue;
        uint32_t incl = 0;
        if (tid < 256) {
            incl = warp_incl_scan(tot);
            if (lane == 31) s_part[warp] = incl;
        }
        __syncthreads();
        if (tid < 256) {
            uint32_t at = incl - tot;
            for (unsigned w = 0; w < warp; ++w) at += s_part[w];
            for (int w = 0; w < kWarps; ++w) {
                const uint32_t c = s_cnt[w * 256 + tid];
                s_cnt[w * 256 + tid] = at;
                at += c;
            }
        }
        __syncthreads();
        for (uint32_t g = r0; g < r1; g += 32) {
            const bool have = g + lane < r1;
            const uint32_t k = have ? src[g + lane] : 0u;
            const uint32_t d = have ? (k >> shift) & 255u : 256u + lane;  // absent lanes match no one
            const uint32_t same = __match_any_sync(kFull, d);
            const uint32_t below = __popc(same & ((1u << lane) - 1u));
            uint32_t at = 0;
            if (have) at = cnt[d];
            __syncwarp();
            if (have && below == 0) cnt[d] = at + __popc(same);
            __syncwarp();
            if (have) dst[at + below] = k;
        }
        __syncthreads();
        uint32_t *t = src;
        src = dst;
        dst = t;
    }
    __syncthreads();  // key_bits may be 0 (all keys 0)
    // first of each run of equal keys; in global memory an odd number of
    // passes leaves the sorted keys in ukeys itself, so they go back first
    if (!local && src != keys + b) {
        for (uint32_t i = tid; i < n; i += THREADS) dst[i] = src[i];
        src = dst;
        __syncthreads();
    }
    uint32_t c = 0;
    for (uint32_t g = r0; g < r1; g += 32) {
        const uint32_t i = g + lane;
        const bool first = i < r1 && (i == 0 || src[i] != src[i - 1]);
        c += __popc(__ballot_sync(kFull, first));
    }
    if (lane == 0) s_part[warp] = c;
    __syncthreads();
    uint32_t at = 0, total = 0;
    for (int w = 0; w < kWarps; ++w) {
        if (w == int(warp)) at = total;
        total += s_part[w];
    }
    for (uint32_t g = r0; g < r1; g += 32) {
        const uint32_t i = g + lane;
        const bool first = i < r1 && (i == 0 || src[i] != src[i - 1]);
        const uint32_t m = __ballot_sync(kFull, first);
        if (first) ukeys[b + at + __popc(m & ((1u << lane) - 1u))] = src[i];
        at += __popc(m);
    }
    if (tid == 0) *ucount = total;
}

// At most 32 keys, one per lane of a warp: each different key's place is the
// number of different keys below it (140,000 queries of 2 keys: 397 us a call,
// 955 with the block's passes over 16-bit keys).
__device__ __forceinline__ void sort_few(const uint32_t *keys, uint32_t n, uint32_t *ukeys, uint32_t *ucount, unsigned lane) {
    const uint32_t k = lane < n ? keys[lane] : 0u;
    const uint32_t live = __ballot_sync(kFull, lane < n);
    const uint32_t same = __match_any_sync(kFull, k) & live;
    const bool first = lane < n && lane == (unsigned)__ffs(same) - 1u;
    const uint32_t firsts = __ballot_sync(kFull, first);
    uint32_t at = 0;
    for (uint32_t m = firsts; m; m &= m - 1) at += __shfl_sync(kFull, k, __ffs(m) - 1) < k ? 1u : 0u;
    if (first) ukeys[at] = k;
    if (lane == 0) *ucount = __popc(firsts);
}

// long_list: [0] number of long queries (zeroed by the caller), [1 ..] the queries.
__global__ void k_long_list(const uint64_t *__restrict__ qoff, uint32_t nq, uint32_t *__restrict__ long_list) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < nq && qoff[q + 1] - qoff[q] > kSortSmallKeys) long_list[1 + atomicAdd(&long_list[0], 1u)] = q;
}

__global__ void __launch_bounds__(kSortSmallThreads) k_unique_sort(uint32_t *keys, const uint64_t *__restrict__ qoff,
                                                                   uint32_t *ukeys, uint32_t *__restrict__ ucount,
                                                                   int key_bits) {
    const uint32_t q = blockIdx.x;
    const uint64_t b = qoff[q], n = qoff[q + 1] - b;  // a query's keys are counted in 32 bits
    if (n > kSortSmallKeys) return;
    if (n <= 32) {
        if (threadIdx.x < 32) sort_few(keys + b, uint32_t(n), ukeys + b, &ucount[q], threadIdx.x);
        return;
    }
    sort_query<kSortSmallThreads, kSortSmallKeys>(keys, b, uint32_t(n), ukeys, &ucount[q], key_bits);
}

__global__ void __launch_bounds__(kSortLargeThreads) k_unique_sort_long(uint32_t *keys, const uint64_t *__restrict__ qoff,
                                                                        uint32_t *ukeys, uint32_t *__restrict__ ucount,
                                                                        const uint32_t *long_list, int key_bits) {
    const uint32_t count = long_list[0];
    for (uint32_t i = blockIdx.x; i < count; i += gridDim.x) {
        const uint32_t q = long_list[1 + i];
        const uint64_t b = qoff[q];
        sort_query<kSortLargeThreads, kSortLargeKeys>(keys, b, uint32_t(qoff[q + 1] - b), ukeys, &ucount[q], key_bits);
        __syncthreads();  // the shared buffers are rewritten for the next query
    }
}

__global__ void k_compact(const uint32_t *__restrict__ ukeys, const uint64_t *__restrict__ qoff,
                          const uint64_t *__restrict__ uoff, uint32_t nq, uint32_t *__restrict__ out) {
    const uint32_t q = blockIdx.x;
    if (q >= nq) return;
    const uint64_t src = qoff[q], dst = uoff[q], n = uoff[q + 1] - uoff[q];
    // four loads in flight per thread
    uint64_t i = threadIdx.x;
    for (; i + 3 * blockDim.x < n; i += 4 * blockDim.x) {
        uint32_t v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = ukeys[src + i + u * blockDim.x];
#pragma unroll
        for (int u = 0; u < 4; ++u) out[dst + i + u * blockDim.x] = v[u];
    }
    for (; i < n; i += blockDim.x) out[dst + i] = ukeys[src + i];
}

// Whether match_unique marks bitmaps: the key space fits one, and what they
// move is worth it.  A bitmap's way out and back costs by its words, sorting
// by the keys, and a warp's sort of up to 32 keys next to nothing.  Calls of
// 20,000 queries (us, bitmaps and sorted): 2 keys each in 256 words 148 and
// 160, in 1,024 194 and 159, in 2,048 228 and 158; 50 keys in 1,024 228 and
// 261; 100 in 2,048 302 and 286, 200 313 and 324; 500 in 4,096 480 and 497;
// 500 in 6,250 606 and 495, 1,000 682 and 735; 1,000 in 10,938 941 and 742,
// 2,000 1,080 and 1,210.  Bitmaps of up to 32 MB stay in L2: 2,000 queries
// of 50 keys in 2,048 words 113 and 117.
inline bool unique_by_bitmap(uint32_t max_key, uint32_t nq, uint64_t keys) {
    const uint64_t words = (max_key >> 5) + 1, all_words = nq * words;
    if (words > kBitmapMaxWords) return false;
    if (words < 1024 || all_words < (uint64_t(8) << 20)) return true;
    if (keys <= uint64_t(nq) * 32) return false;
    return words < 2048 || keys * (words < 4096 ? 20 : 8) >= all_words;
}

inline void launch_unique_mark(const uint32_t *keys, const uint64_t *qoff, uint32_t nq, uint64_t n_keys, uint32_t words,
                               uint32_t *bitmaps, uint32_t *ucount, int sm_count, cudaStream_t st) {
    // the bitmap and the count may together exceed the default 48 KB
    TM_CUDA(cudaFuncSetAttribute(k_unique_mark, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kBitmapMaxWords * 4)));
    // no more threads than have four stores of the bitmap's words or two
    // loads of four keys each to make (140,000 queries of 100 keys in 32 words,
    // with the read-out's: 669 us a call with 256 and eight warps, 320 so)
    unsigned threads = nq <= 4u * unsigned(sm_count) ? 1024 : 256;
    const uint64_t busy = std::max<uint64_t>(bitmap_stride(words) / 16, n_keys / nq / 8);
    while (threads > 32 && threads / 2 >= busy) threads /= 2;
    k_unique_mark<<<nq, threads, bitmap_stride(words) * 4, st>>>(keys, qoff, words, bitmaps, ucount);
    TM_CHECK_LAUNCH();
}

inline void launch_unique_expand(const uint32_t *bitmaps, const uint64_t *uoff, uint32_t nq, uint32_t words, uint32_t *out,
                                 cudaStream_t st) {
    // a warp for each round of 64 words
    if (words > 256) k_unique_expand<8><<<nq, 256, 0, st>>>(bitmaps, uoff, words, out);
    else if (words > 128) k_unique_expand<4><<<nq, 128, 0, st>>>(bitmaps, uoff, words, out);
    else if (words > 64) k_unique_expand<2><<<nq, 64, 0, st>>>(bitmaps, uoff, words, out);
    else k_unique_expand<1><<<nq, 32, 0, st>>>(bitmaps, uoff, words, out);
    TM_CHECK_LAUNCH();
}

// Sorts every query's keys and leaves the different ones in ukeys[qoff ..).
// long_list: scratch of nq + 1 words.  The long queries are sorted beside the
// others where the caller has a stream for them (2,000 queries of 1,070 keys:
// the two kernels take 84 and 94 us, one after the other before).
inline void launch_unique_sort(uint32_t *keys, const uint64_t *qoff, uint32_t nq, uint32_t *ukeys, uint32_t *ucount,
                               uint32_t *long_list, uint32_t max_key, int sm_count, cudaStream_t st,
                               SideStream *side = nullptr) {
    int key_bits = 0;
    while (key_bits < 32 && (max_key >> key_bits)) ++key_bits;
    constexpr int small = kSortSmem<kSortSmallThreads, kSortSmallKeys>, large = kSortSmem<kSortLargeThreads, kSortLargeKeys>;
    TM_CUDA(cudaFuncSetAttribute(k_unique_sort_long, cudaFuncAttributeMaxDynamicSharedMemorySize, large));
    TM_CUDA(cudaMemsetAsync(long_list, 0, sizeof(uint32_t), st));
    k_long_list<<<blocks_for(nq, 256), 256, 0, st>>>(qoff, nq, long_list);
    TM_CHECK_LAUNCH();
    cudaStream_t beside = side ? side->fork(st) : st;
    k_unique_sort_long<<<std::min<uint32_t>(nq, uint32_t(sm_count)), kSortLargeThreads, large, beside>>>(
        keys, qoff, ukeys, ucount, long_list, key_bits);
    TM_CHECK_LAUNCH();
    k_unique_sort<<<nq, kSortSmallThreads, small, st>>>(keys, qoff, ukeys, ucount, key_bits);
    TM_CHECK_LAUNCH();
    if (side) side->join(st);
}

// Copies na words at a, nb at b, then nc at c, into mapped pinned host memory
// (dst is its device view).  Used for the few numbers the host needs in the
// middle of a batch (queue sizes, pair and key totals).
__global__ void k_readback(const uint32_t *__restrict__ a, uint32_t na, const uint32_t *__restrict__ b, uint32_t nb,
                           const uint32_t *__restrict__ c, uint32_t nc, uint32_t *__restrict__ dst) {
    const uint32_t n = na + nb + nc;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        dst[i] = i < na ? a[i] : i < na + nb ? b[i - na] : c[i - na - nb];
}

// Keys narrowed to 16 bits for the trip to the host (tables whose largest
// key is below 65,536); the host widens them back.
__global__ void k_narrow16(const uint32_t *__restrict__ in, uint64_t n, uint16_t *__restrict__ out) {
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i * 4 < n; i += stride) {
        if (i * 4 + 4 <= n && (reinterpret_cast<uintptr_t>(in) & 15) == 0) {
            const uint4 v = reinterpret_cast<const uint4 *>(in)[i];
            uint2 w;
            w.x = (v.x & 0xFFFFu) | (v.y << 16);
            w.y = (v.z & 0xFFFFu) | (v.w << 16);
            reinterpret_cast<uint2 *>(out)[i] = w;
        } else {
            for (uint64_t k = i * 4; k < n && k < i * 4 + 4; ++k) out[k] = uint16_t(in[k]);
        }
    }
}

}  // namespace
}  // namespace tmb
