// How large the matcher's optional or guessed device buffers are made: plain
// rules over sizes, apart from the device so that they can be run without one.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace tmb {

constexpr size_t kRecordBytes = 16;               // one hit record
constexpr size_t kSpareRecords = size_t(1) << 20;  // of a first buffer, beside those per query
// Hit records per query that a buffer is made for ahead of its first batch.
// A batch that has more runs again with a larger buffer, at twice the time,
// which is what the first batches of an engine did on ten million filters:
// there a query makes 3,350 records (446,000 tiles), 690 on a million (44,000),
// 950 on two million skewed ones (98,000).
constexpr size_t kLeastRecords = 512, kMostRecords = 4608;
constexpr size_t records_per_query(uint32_t n_tiles) {
    return kLeastRecords + n_tiles / 128 < kMostRecords ? kLeastRecords + n_tiles / 128 : kMostRecords;
}
// A guess may take this share of the device memory that is free with the
// buffer given back: the keys, whose size is known and must be had, come after.
constexpr size_t kGuessShare = 8;
// What a budget (bytes, 0: none) leaves to a buffer that may take 1 / share of
// it: a batch's guesses and conveniences must leave room for its records and
// keys, which the number of queries admitted is reckoned from.
constexpr size_t budget_share(size_t budget, size_t share) { return budget ? budget / share : ~size_t(0); }
constexpr size_t kGuessBudgetShare = 2;   // hit records ahead of the batch
constexpr size_t kQueueBudgetShare = 4;   // queues allocated before they are counted
constexpr size_t kBitmapBudgetShare = 4;  // match_unique's bitmaps

// What the batches of one scratch have shown of its table's hit records.
struct RecordHistory {
    uint32_t n_tiles = 0;                  // the table they were matched on
    uint64_t queries = 0, records = 0;     // seen
    size_t ceiling = ~size_t(0);           // records that a guess may not exceed any more

    void seen(uint32_t nq, uint64_t n) {
        queries += nq;
        records += n;
        if (queries > (uint64_t(1) << 20)) {  // later batches count more
            queries /= 2;
            records /= 2;
        }
    }
    // Records expected of nq queries: the table's guess, which weighs as much
    // as 64 queries, and what was seen, with a margin of a quarter.
    size_t expected(uint32_t nq, uint32_t tiles) {
        if (tiles != n_tiles) {
            *this = RecordHistory();
            n_tiles = tiles;
        }
        const double guess = double(records_per_query(tiles));
        const double per_query = (64.0 * guess + 1.25 * double(records)) / (64.0 + double(queries));
        return size_t(double(nq) * std::min(guess, per_query));
    }
};

// Makes the record buffer ready for a batch: never smaller than it is (at
// first kLeastRecords a query and the spare ones), larger where the batch is
// expected to need it and a share of the free memory, and of the budget,
// allows.  What was refused once, by that share or by the allocator, is not
// tried again: every further try would free the buffer that serves, fail, and
// make the small one again, with the subset test run twice after it (65,536
// queries without matches on ten million filters with 3 GiB free: 2,970 us or
// more for every call, 170 since).  free_bytes() is asked only when the buffer
// would grow.
template <class Buf, class FreeBytes>
void reserve_records(Buf &recs, RecordHistory &h, uint32_t nq, uint32_t n_tiles, size_t budget, FreeBytes free_bytes) {
    const size_t held = recs.p ? recs.cap : 0;
    const size_t least = held ? held : size_t(nq) * kLeastRecords + kSpareRecords;
    size_t want = std::min(h.expected(nq, n_tiles), h.ceiling);
    want = std::min(want, budget_share(budget, kGuessBudgetShare) / kRecordBytes);
    if (want > least) {
        const size_t room = (free_bytes() / kRecordBytes + held) / kGuessShare;
        if (want > room) h.ceiling = want = room;
    }
    if (want > least) {
        if (recs.try_reserve(want)) return;
        h.ceiling = least;
    }
    recs.reserve(least);
}

// Makes the queues and slices ready by their bound, which saves the wait for
// their exact sizes: when that takes no more than `limit` bytes and can be had.
// False: they are to be made by their exact sizes, which may fit where the
// bound does not.  A refused size is not tried again.
template <class Queue, class Slices>
bool reserve_ahead(Queue &queue, size_t queue_len, Slices &slices, size_t slice_len, size_t bytes, size_t limit, size_t &refused) {
    if (bytes > limit || bytes >= refused) return false;
    if (queue.try_reserve(queue_len) && slices.try_reserve(slice_len)) return true;
    queue.release();  // what it got would be missing beside
    refused = bytes;
    return false;
}

// Whether a budget allows match_unique's bitmaps: never more than its share, or
// than sorting, which takes a second buffer for the keys, would take.
constexpr bool bitmaps_allowed(size_t bitmap_bytes, size_t key_bytes, size_t budget) {
    return bitmap_bytes <= std::max(key_bytes, budget_share(budget, kBitmapBudgetShare));
}

// Makes room for match_unique's bitmaps (words of 4 bytes); false when there is
// none: they may take 1 GiB, or a share of the free memory, and sorting does
// without.  A size that was refused is not tried again (refused: kept beside
// the buffer).
constexpr size_t kBitmapBytesAnyway = size_t(1) << 30;
template <class Buf, class FreeBytes>
bool reserve_bitmaps(Buf &buf, size_t words, size_t &refused, FreeBytes free_bytes) {
    if (buf.p && words <= buf.cap) return true;
    if (words >= refused) return false;
    const size_t held = buf.p ? buf.cap : 0;
    if ((words * 4 <= kBitmapBytesAnyway || words * 4 <= (free_bytes() + held * 4) / kGuessShare) && buf.try_reserve(words))
        return true;
    refused = words;
    return false;
}

}  // namespace tmb
