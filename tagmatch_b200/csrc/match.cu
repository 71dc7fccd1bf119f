// Batched subset matching on one device.
//
// The reference routes each query on CPU threads to every partition whose
// mask is a subset of the query (front_end.cc:465-477), queues it per
// partition, ships full queues of 256 queries to the GPU
// (front_end.cc:350-376, back_end.cc:243-302) where three_phase_matching
// (gpu.cu:60-607) tests one filter per thread against the batch held in
// constant memory and appends every hit with a global atomic
// (gpu.cu:53-58); the host then turns (query, filter) hits into keys
// (back_end.cc:288-302) and sorts/uniques them for match_unique
// (tagmatch_query.hh:99-119).
//
// Here the whole path runs on the device for a batch of queries:
//   k_route      one thread per query tests the partition masks (held in
//                shared memory): a vote per (partition, 32 queries) gives
//                the routing matrix, a bit per (partition, query), and the
//                partitions' counts;
//   k_plan       queue, chunk and work item offsets from the counts; work
//                items = (partition, group of four 256-query chunks, segment
//                of the partition's tiles), partitions in id order or in the
//                order the learned cost model gives;
//   k_fill_queues  each partition's queue from its row of the matrix:
//                records of 32 bytes (6 query words, query id, pad) and, per
//                256-query chunk, bit-sliced "lacks bit b" masks: Z[b] bit j
//                set when query j of the chunk lacks bit b (192 x 256 bits,
//                bit transposes of the query words);
//   k_match      persistent CTAs take items from an atomic counter.  Each
//                item's query records are staged into shared memory by bulk
//                TMA copies (cp.async.bulk + mbarrier); the buffers are
//                released by per-warp mbarrier arrivals.  A warp selects the
//                candidate queries of one tile of <= 32 filters (or of
//                several, for items of few queries) by OR-ing the slices of
//                bits that all the tile's filters hold, one 32-query word
//                per lane; the candidates are tested either two or one per
//                lane against the tile's filters broadcast from shared
//                memory, or, when they are few, four at a time against the
//                tile held one filter per lane (6 LOP3s per (query, filter)
//                either way); each (query, tile) with a hit becomes a
//                (query, tile, hit mask, key count) record, staged per warp
//                in shared memory and flushed with one global atomic, which
//                is when its keys are counted and added to the query's
//                total;
//   k_key_fill   after a prefix sum of the query totals: one cursor atomic
//                per record (per query and block of records for batches of
//                few queries); the runs of adjacent hit bits of a warp's 64
//                records (one key range each) are numbered and copied 32 at
//                a time by the whole warp;
//   k_unique_*   match_unique: per-query bitmap, read out in order (small
//                key spaces), or per-query block radix sort + unique.
// Result overflow is exact: the record buffer is regrown and the batch re-run
// (the reference truncates silently at 4,194,304 hits, gpu.cu:55).
#include "match_kernels.cuh"
#include <cstdio>
#include <cstring>
#include <cstdlib>

namespace tmb {

MatchScratch &MatchScratch::operator=(MatchScratch &&o) noexcept {
    if (this == &o) return *this;
    queries = std::move(o.queries);
    zeroed = std::move(o.zeroed);
    rows = std::move(o.rows);
    part_off = std::move(o.part_off);
    queue = std::move(o.queue);
    item_off = std::move(o.item_off);
    chunk_off = std::move(o.chunk_off);
    slices = std::move(o.slices);
    work = std::move(o.work);
    keys16 = std::move(o.keys16);
    recs = std::move(o.recs);
    qoff = std::move(o.qoff);
    keys = std::move(o.keys);
    ucount = std::move(o.ucount);
    uoff = std::move(o.uoff);
    ukeys = std::move(o.ukeys);
    readback = std::move(o.readback);
    part_order = std::move(o.part_order);
    d_part_order = std::move(o.d_part_order);
    record_items = o.record_items;
    item_stats = std::move(o.item_stats);
    h_item_stats = std::move(o.h_item_stats);
    for (int i = 0; i < 2 * ScanScratch::kLevels; ++i) scr.levels[i] = std::move(o.scr.levels[i]);
    side.swap(o.side);
    sm_count = o.sm_count;
    rec_history = o.rec_history;
    bitmaps_refused = o.bitmaps_refused;
    ahead_refused = o.ahead_refused;
    row_words = o.row_words;
    seg_tiles = o.seg_tiles;
    seg_exact = o.seg_exact;
    budget = o.budget;
    profile = o.profile;
    if (ev_begin) cudaEventDestroy(ev_begin);
    if (ev_end) cudaEventDestroy(ev_end);
    ev_begin = o.ev_begin;
    ev_end = o.ev_end;
    o.ev_begin = o.ev_end = nullptr;
    return *this;
}

// Estimated cost of one 4-candidate trip of the subset test's
// lane-per-filter loop, against which the lane-per-query pass is weighed
// for each tile (TM_FPL_TRIP_COST overrides it; results do not depend on
// it; items of more than 512 queries always take the pass).  Measured on
// 524,288 queries and ten million filters with 1,024-query work items: flat
// from 75 to 150, worse below (45: +9%).
uint32_t fpl_trip_cost() {
    static const uint32_t v = [] {
        const char *e = std::getenv("TM_FPL_TRIP_COST");
        return e ? uint32_t(std::strtoul(e, nullptr, 10)) : 90u;
    }();
    return v;
}

const uint16_t *narrow_keys(const uint32_t *d_keys, uint64_t n, MatchScratch &s, cudaStream_t st) {
    s.keys16.reserve(std::max<uint64_t>(n, 1) + 8);
    if (n) {
        const unsigned blocks = unsigned(std::min<uint64_t>((n / 4 + 255) / 256 + 1, 148 * 16));
        k_narrow16<<<blocks, 256, 0, st>>>(d_keys, n, s.keys16.p);
        TM_CHECK_LAUNCH();
    }
    return s.keys16.p;
}

// Reads na words at a, nb at b and nc at c (device memory) into s.readback
// and waits for them: a kernel writes them to mapped host memory, so the
// read does not wait for copies that other streams have queued on the copy
// engines (the host pipeline keeps multi-GB result copies in flight while
// the next batch is matched).
const uint32_t *read_back(MatchScratch &s, const void *a, uint32_t na, const void *b, uint32_t nb, const void *c, uint32_t nc,
                          cudaStream_t st) {
    const uint32_t n = na + nb + nc;
    s.readback.reserve(n);
    const unsigned blocks = std::min(64u, (n + 255) / 256);
    k_readback<<<std::max(blocks, 1u), 256, 0, st>>>(static_cast<const uint32_t *>(a), na, static_cast<const uint32_t *>(b), nb,
                                                     static_cast<const uint32_t *>(c), nc, s.readback.d);
    TM_CHECK_LAUNCH();
    TM_CUDA(cudaStreamSynchronize(st));
    return s.readback.h;
}

// Queues and slices are allocated by their exact sizes, which takes a wait
// for the partitions' counts in the middle of the batch; when even every
// query in every partition would need no more than this, that is allocated
// and the wait saved (it is paid by small batches: about 10 us of 180 for
// one query).
constexpr size_t kQueueAheadBytes = size_t(256) << 20;

size_t free_device_bytes() {
    size_t free_bytes = 0, all_bytes = 0;
    TM_CUDA(cudaMemGetInfo(&free_bytes, &all_bytes));
    return free_bytes;
}

static_assert(sizeof(HitRec) == kRecordBytes, "the record buffer is sized in records");

MatchScratch::~MatchScratch() {
    if (ev_begin) cudaEventDestroy(ev_begin);
    if (ev_end) cudaEventDestroy(ev_end);
}

void match_batch(const DevTable &t, const uint32_t *d_queries, uint32_t nq, bool unique, MatchScratch &s,
                 const uint64_t **d_offsets, const uint32_t **d_keys, uint64_t *n_keys, BatchStats *stats,
                 cudaStream_t st, cudaEvent_t match_begin, cudaEvent_t match_end) {
    if (s.sm_count == 0) {
        int dev;
        TM_CUDA(cudaGetDevice(&dev));
        TM_CUDA(cudaDeviceGetAttribute(&s.sm_count, cudaDevAttrMultiProcessorCount, dev));
    }
    const uint32_t P = t.n_parts;
    BatchStats bs;
    s.qoff.reserve(size_t(nq) + 1);
    if (nq == 0 || P == 0 || t.n_tiles == 0) {
        TM_CUDA(cudaMemsetAsync(s.qoff.p, 0, (size_t(nq) + 1) * sizeof(uint64_t), st));
        TM_CUDA(cudaStreamSynchronize(st));
        *d_offsets = s.qoff.p;
        *d_keys = s.keys.p;
        *n_keys = 0;
        if (match_begin) TM_CUDA(cudaEventRecord(match_begin, st));
        if (match_end) TM_CUDA(cudaEventRecord(match_end, st));
        if (stats) *stats = bs;
        return;
    }
    // ---- routing ----
    // everything that starts at zero, cleared together
    const uint32_t groups = route_groups(nq);
    const size_t n_zero = 8 + size_t(P) * (1 + groups) + 2 * size_t(nq);
    s.zeroed.reserve(n_zero);
    unsigned long long *counters = reinterpret_cast<unsigned long long *>(s.zeroed.p);
    uint32_t *qkeys = s.zeroed.p + 8, *qcursor = qkeys + nq, *part_count = qcursor + nq, *group_count = part_count + P;
    TM_CUDA(cudaMemsetAsync(s.zeroed.p, 0, n_zero * sizeof(uint32_t), st));
    uint32_t window = route_window(P, nq, s.row_words);
    while (window > 32 && !s.rows.try_reserve(size_t(window) * route_row_words(nq))) {
        s.row_words /= 2;  // smaller windows where the device is short of memory
        window = route_window(P, nq, s.row_words);
    }
    s.rows.reserve(size_t(window) * route_row_words(nq));
    const uint32_t windows = (P + window - 1) / window;
    for (uint32_t p0 = 0; p0 < P; p0 += window)
        launch_route(true, d_queries, nq, t, p0, std::min(P, p0 + window), s.rows.p, part_count, group_count, st);
    // ---- plan: queue positions, chunks and work items ----
    const bool ordered = s.part_order.size() == P;
    if (ordered) {
        s.d_part_order.reserve(P);
        TM_CUDA(cudaMemcpyAsync(s.d_part_order.p, s.part_order.data(), size_t(P) * 4, cudaMemcpyHostToDevice, st));
    }
    const uint32_t *order = ordered ? s.d_part_order.p : nullptr;
    s.part_off.reserve(size_t(P) + 1);
    s.chunk_off.reserve(size_t(P) + 1);
    s.item_off.reserve(size_t(P) + 4);
    // batches whose items are timed for the cost model take the tiles per item
    // as they are set, the model learns their effect; and so do those for
    // which it chose them
    const uint32_t least = least_seg(nq);
    const uint32_t want_items = s.record_items || s.seg_exact ? 0 : uint32_t(s.sm_count) * 4 * kItemsPerCta;
    k_plan<<<1, kPlanThreads, 0, st>>>(part_count, t.part_tile_begin.p, order, P, s.seg_tiles, least, want_items, s.part_off.p,
                                       s.chunk_off.p, s.item_off.p, s.item_off.p + P + 1);
    TM_CHECK_LAUNCH();
    // the host's copy of the plan, once the counts are back
    uint32_t items = 0, chunks = 0;
    auto host_plan = [&](const uint32_t *counts) {
        s.h_part_count.assign(counts, counts + P);
        s.h_item_off.resize(size_t(P) + 1);
        uint32_t seg = s.seg_tiles;  // as k_plan chooses it
        for (int h = 0; want_items && h < kSegHalvings; ++h) {
            uint64_t total = 0;
            for (uint32_t p = 0; p < P; ++p)
                total += part_items(counts[p], t.h_part_tiles[p + 1] - t.h_part_tiles[p], halved_seg(s.seg_tiles, h, least));
            if (total >= want_items) break;
            seg = halved_seg(s.seg_tiles, h + 1, least);
        }
        for (uint32_t pos = 0; pos < P; ++pos) {
            bs.routed += counts[pos];
            bs.dense += uint64_t(counts[pos]) * t.h_part_size[pos];
            chunks += (counts[pos] + kChunk - 1) / kChunk;
            // work items in the queue order: partition id order, or the order
            // the learned cost model gives (most expensive items first)
            const uint32_t p = ordered ? s.part_order[pos] : pos;
            s.h_item_off[pos] = items;
            // an item: kItemChunks chunks of the partition x one tile segment
            items += part_items(counts[p], t.h_part_tiles[p + 1] - t.h_part_tiles[p], seg);
        }
        s.h_item_off[P] = items;
        bs.items = items;
    };
    size_t queue_len = size_t(nq) * P, slice_len = size_t(P) * blocks_for(nq, kChunk);
    const bool ahead = !s.record_items &&
                       reserve_ahead(s.queue, queue_len * 2, s.slices, slice_len * kSliceWords,
                                     queue_len * kQueueWords * 4 + slice_len * kSliceWords * 4,
                                     std::min(kQueueAheadBytes, budget_share(s.budget, kQueueBudgetShare)), s.ahead_refused);
    if (!ahead) {
        host_plan(read_back(s, part_count, P, nullptr, 0, nullptr, 0, st));
        queue_len = bs.routed;
        slice_len = chunks;
    }
    s.queue.reserve(std::max<size_t>(queue_len, 1) * 2);
    uint4 *queue_lo = s.queue.p, *queue_hi = s.queue.p + queue_len;
    s.slices.reserve(std::max<size_t>(slice_len, 1) * kSliceWords);
    launch_fill_queues(d_queries, nq, t, window, s.rows.p, part_count, group_count, s.part_off.p, s.chunk_off.p, queue_lo,
                       queue_hi, s.slices.p, st);
    // route, queues (both again per window), plan, match, scan, readback
    bs.launches += windows * (windows > 1 ? 3 : 2) + 3 + scan_launches(nq) + (ahead ? 0u : 1u);
    // ---- match (regrow and re-run on pair overflow) ----
    reserve_records(s.recs, s.rec_history, nq, t.n_tiles, s.budget, free_device_bytes);
    unsigned long long hc[4] = {0, 0, 0, 0};
    uint64_t total = 0;
    for (int attempt = 0;; ++attempt) {
        // counters and the per-query key totals, which the subset test sums
        // itself, are zero at first
        if (attempt) TM_CUDA(cudaMemsetAsync(s.zeroed.p, 0, (8 + size_t(nq)) * sizeof(uint32_t), st));
        static const bool work_counters = std::getenv("TM_WORK_COUNTERS") != nullptr;
        if (work_counters) {
            s.work.reserve(8);
            TM_CUDA(cudaMemsetAsync(s.work.p, 0, 8 * sizeof(unsigned long long), st));
        }
        if (s.record_items) {
            s.item_stats.reserve(2 * size_t(std::max<uint32_t>(items, 1)));
            TM_CUDA(cudaMemsetAsync(s.item_stats.p, 0, 2 * size_t(items) * sizeof(unsigned long long), st));
        }
        MatchArgs a{t.tile_words.p, t.tile_info.p, t.tile_keys.p, t.slot_key_off.p, t.part_tile_begin.p, part_count,
                    s.part_off.p, s.item_off.p, s.chunk_off.p, queue_lo, queue_hi, s.slices.p, P, s.item_off.p + P + 1, counters,
                    s.recs.p, (unsigned long long)s.recs.cap, qkeys, fpl_trip_cost(), order, s.record_items ? s.item_stats.p : nullptr,
                    work_counters ? s.work.p : nullptr};
        if (match_begin && attempt == 0) TM_CUDA(cudaEventRecord(match_begin, st));
        if (s.profile) {
            if (!s.ev_begin) {
                TM_CUDA(cudaEventCreate(&s.ev_begin));
                TM_CUDA(cudaEventCreate(&s.ev_end));
            }
            TM_CUDA(cudaEventRecord(s.ev_begin, st));
        }
        if (work_counters) launch_match<true>(a, unsigned(s.sm_count) * 4, st);
        else launch_match<false>(a, unsigned(s.sm_count) * 4, st);
        TM_CHECK_LAUNCH();
        if (s.profile) TM_CUDA(cudaEventRecord(s.ev_end, st));
        if (match_end) TM_CUDA(cudaEventRecord(match_end, st));
        exclusive_scan<uint32_t, uint64_t>(qkeys, s.qoff.p, nq, s.scr, st);
        const uint32_t *rb = read_back(s, counters, 8, s.qoff.p + nq, 2, part_count, ahead && !attempt ? P : 0u, st);
        std::memcpy(hc, rb, sizeof(hc));
        std::memcpy(&total, rb + 8, sizeof(total));
        if (ahead && !attempt) host_plan(rb + 10);
        if (hc[2]) throw Error(TM_ERR_TIMEOUT, "match kernel: bounded wait for the query copy expired");
        if (work_counters) {
            unsigned long long w[8];
            TM_CUDA(cudaMemcpy(w, s.work.p, sizeof(w), cudaMemcpyDeviceToHost));
            std::fprintf(stderr,
                         "[tm work] queries %u tile_visits %llu query_passes %llu candidates %llu filter_trips %llu "
                         "items %llu query_groups %llu query_lanes %llu small_query_visits %llu records %llu pairs %llu\n",
                         nq, w[0], w[1], w[2], w[3], w[4], w[5], w[6], w[7], hc[1], hc[3]);
        }
        if (s.profile) {
            float ms = 0.f;
            TM_CUDA(cudaEventElapsedTime(&ms, s.ev_begin, s.ev_end));
            bs.match_ms += ms;
        }
        if (hc[1] <= s.recs.cap) break;
        if (attempt >= 3) throw Error(TM_ERR_INTERNAL, "hit record buffer regrowth did not converge");
        s.recs.reserve(size_t(hc[1] + hc[1] / 4 + 1024));
        bs.retries++;
    }
    bs.records = hc[1];
    s.rec_history.seen(nq, hc[1]);
    if (s.record_items) {
        s.h_item_stats.resize(2 * size_t(items));
        if (items)
            TM_CUDA(cudaMemcpyAsync(s.h_item_stats.data(), s.item_stats.p, 2 * size_t(items) * sizeof(unsigned long long),
                                    cudaMemcpyDeviceToHost, st));
    }
    // ---- keys ----
    // fill; each retry: match, scan, readback
    bs.launches += 1 + (2 + scan_launches(nq)) * uint32_t(bs.retries);
    bs.pairs = hc[3];
    s.keys.reserve(std::max<uint64_t>(total, 1));
    bs.key_bytes = total * 4;
    launch_key_fill(t, s.recs.p, counters, hc[1], total, s.qoff.p, qcursor, nq, s.keys.p, s.sm_count, st);
    if (!unique) {
        TM_CUDA(cudaStreamSynchronize(st));
        *d_offsets = s.qoff.p;
        *d_keys = s.keys.p;
        *n_keys = total;
        bs.keys = total;
        if (stats) *stats = bs;
        return;
    }
    // ---- match_unique ----
    s.ucount.reserve(nq);
    s.uoff.reserve(size_t(nq) + 1);
    const uint32_t words = (t.max_key >> 5) + 1;
    const size_t bitmap_words = size_t(nq) * bitmap_stride(words);
    const bool bitmaps = unique_by_bitmap(t.max_key, nq, total) && bitmaps_allowed(bitmap_words * 4, total * 4, s.budget) &&
                         reserve_bitmaps(s.ukeys, bitmap_words, s.bitmaps_refused, free_device_bytes);
    bs.key_bytes += bitmaps ? bitmap_words * 4 : total * 4;
    if (bitmaps) {
        launch_unique_mark(s.keys.p, s.qoff.p, nq, total, words, s.ukeys.p, s.ucount.p, s.sm_count, st);
        exclusive_scan<uint32_t, uint64_t>(s.ucount.p, s.uoff.p, nq, s.scr, st);
        launch_unique_expand(s.ukeys.p, s.uoff.p, nq, words, s.keys.p, st);
        bs.launches += 3 + scan_launches(nq);  // mark, expand, readback, scan
    } else {
        s.ukeys.reserve(std::max<uint64_t>(total, 1));
        // the offsets' buffer holds the list of long queries until the scan
        launch_unique_sort(s.keys.p, s.qoff.p, nq, s.ukeys.p, s.ucount.p, reinterpret_cast<uint32_t *>(s.uoff.p), t.max_key,
                           s.sm_count, st, &s.side);
        exclusive_scan<uint32_t, uint64_t>(s.ucount.p, s.uoff.p, nq, s.scr, st);
        // compact into s.keys (unique prefix of every segment is <= its length)
        k_compact<<<nq, 256, 0, st>>>(s.ukeys.p, s.qoff.p, s.uoff.p, nq, s.keys.p);
        TM_CHECK_LAUNCH();
        bs.launches += 5 + scan_launches(nq);  // list, two sorts, compact, readback, scan
    }
    uint64_t utotal = 0;
    std::memcpy(&utotal, read_back(s, s.uoff.p + nq, 2, nullptr, 0, nullptr, 0, st), sizeof(uint64_t));
    *d_offsets = s.uoff.p;
    *d_keys = s.keys.p;
    *n_keys = utotal;
    bs.keys = utotal;
    if (stats) *stats = bs;
}

}  // namespace tmb
