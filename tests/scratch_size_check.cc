// The matcher's buffer size rules over an allocator with a limit, no device.
#include "../tagmatch_b200/csrc/scratch_size.hpp"
#include <cstdio>
#include <cstdlib>

#define CHECK(x)                                                   \
    do {                                                           \
        if (!(x)) {                                                \
            std::printf("%s:%d: %s\n", __FILE__, __LINE__, #x);    \
            std::exit(1);                                          \
        }                                                          \
    } while (0)

// A buffer like the device's: growing frees first, and may be refused.
struct Device {
    size_t free_bytes;
    int allocations = 0, refusals = 0;
};
struct Buf {
    Device &dev;
    size_t element;
    void *p = nullptr;
    size_t cap = 0;
    bool try_reserve(size_t n) {
        if (p && n <= cap) return true;
        if (p) n = std::max(n, cap + cap / 2);
        release();
        if (n * element > dev.free_bytes) return ++dev.refusals, false;
        dev.free_bytes -= n * element;
        ++dev.allocations;
        p = this;
        cap = n;
        return true;
    }
    void reserve(size_t n) { CHECK(try_reserve(n)); }
    void release() {
        dev.free_bytes += cap * element;
        p = nullptr;
        cap = 0;
    }
};

static void batch(Buf &b, tmb::RecordHistory &h, uint32_t nq, uint32_t tiles, uint64_t records, int *runs = nullptr,
                  size_t budget = 0) {
    tmb::reserve_records(b, h, nq, tiles, budget, [&] { return b.dev.free_bytes; });
    if (records > b.cap) {
        b.reserve(records + records / 4 + 1024);
        if (runs) ++*runs;
    }
    h.seen(nq, records);
}

int main() {
    const size_t GiB = size_t(1) << 30;
    const uint32_t tiles = 446000, nq = 65536;  // ten million filters
    for (uint64_t per_query : {0, 100, 3350}) {
        for (size_t free_gib : {3, 5, 8, 20, 170}) {
            Device dev{free_gib * GiB};
            Buf b{dev, tmb::kRecordBytes};
            tmb::RecordHistory h;
            if (per_query * nq * 5 / 4 * tmb::kRecordBytes > free_gib * GiB) continue;  // does not fit at all
            int runs = 0;
            batch(b, h, nq, tiles, per_query * nq, &runs);
            // a guess takes no more than its share; what is needed is had
            CHECK(dev.refusals == 0);
            if (!runs) CHECK(b.cap * tmb::kRecordBytes <= std::max(free_gib * GiB / tmb::kGuessShare, (nq * size_t(512) + (1u << 20)) * 16));
            const int allocations = dev.allocations;
            const size_t cap = b.cap;
            for (int i = 0; i < 50; ++i) batch(b, h, nq, tiles, per_query * nq, &runs);
            CHECK(dev.allocations == allocations && b.cap == cap && dev.refusals == 0);
            CHECK(runs == (allocations > 1 ? 1 : 0));
            // a smaller batch leaves the buffer
            batch(b, h, 1, tiles, per_query);
            CHECK(b.cap == cap);
            // with memory to spare the first batch does not run twice
            if (free_gib == 170) CHECK(runs == 0);
        }
    }
    {   // a guess that the allocator refuses all the same is made once
        Device dev{3 * GiB};
        Buf b{dev, tmb::kRecordBytes};
        tmb::RecordHistory h;
        auto all_free = [] { return size_t(170) << 30; };
        tmb::reserve_records(b, h, nq, tiles, 0, all_free);
        CHECK(dev.refusals == 1 && b.cap == nq * size_t(512) + (1u << 20));
        for (int i = 0; i < 5; ++i) tmb::reserve_records(b, h, nq, tiles, 0, all_free);
        CHECK(dev.refusals == 1 && dev.allocations == 1);
    }
    {   // small batches first: later ones are sized by what was seen, not by
        // the table alone, and one query's records are no measure
        Device dev{170 * GiB};
        Buf b{dev, tmb::kRecordBytes};
        tmb::RecordHistory h;
        for (int i = 0; i < 20; ++i) batch(b, h, 1000, tiles, 1000 * 20);
        batch(b, h, 4 * nq, tiles, size_t(4) * nq * 20);
        CHECK(b.cap * 16 < GiB);
        tmb::RecordHistory one;
        one.seen(1, 400000);
        CHECK(one.expected(nq, tiles) <= size_t(nq) * tmb::kMostRecords);
    }
    {   // another table starts over
        tmb::RecordHistory h;
        h.expected(1, tiles);
        h.seen(100000, 0);
        h.ceiling = 5;
        CHECK(h.expected(1000, 128 * 200) == 1000 * 712 && h.ceiling == ~size_t(0));
    }
    for (size_t budget : {size_t(1) << 20, GiB / 4, 16 * GiB}) {  // a lane's budget bounds the guess, not what is needed
        Device dev{170 * GiB};
        Buf b{dev, tmb::kRecordBytes};
        tmb::RecordHistory h;
        const uint32_t n = uint32_t(std::max<size_t>(1, std::min<size_t>(nq, budget / (64 << 10))));
        batch(b, h, n, tiles, size_t(n) * 20, nullptr, budget);
        CHECK(b.cap * 16 <= std::max(budget / 2, (n * size_t(512) + (1u << 20)) * 16));
        batch(b, h, n, tiles, size_t(n) * 5000, nullptr, budget);
        CHECK(b.cap >= size_t(n) * 5000);
        // bitmaps: a quarter of the budget, or what sorting would take
        CHECK(tmb::bitmaps_allowed(budget / 4, 0, budget));
        CHECK(!tmb::bitmaps_allowed(budget / 4 + 1, 0, budget));
        CHECK(tmb::bitmaps_allowed(budget / 4 + 1, budget / 4 + 1, budget));
    }
    CHECK(tmb::bitmaps_allowed(100 * GiB, 0, 0));
    {   // refused bitmaps are not asked for again, smaller ones are
        Device dev{GiB};
        Buf b{dev, 4};
        size_t refused = ~size_t(0);
        auto free_bytes = [&] { return dev.free_bytes; };
        for (int i = 0; i < 5; ++i) {
            CHECK(!tmb::reserve_bitmaps(b, GiB / 4 + 1, refused, free_bytes));  // by the share
            b.reserve(1000);  // the sorting route's buffer
        }
        CHECK(dev.refusals == 0 && dev.allocations == 1);
        dev.free_bytes -= GiB / 2;
        for (int i = 0; i < 5; ++i) {
            CHECK(!tmb::reserve_bitmaps(b, GiB / 4, refused, free_bytes));  // by the allocator
            b.reserve(1000);
        }
        CHECK(dev.refusals == 1 && dev.allocations == 2);
        CHECK(tmb::reserve_bitmaps(b, GiB / 16, refused, free_bytes) && tmb::reserve_bitmaps(b, GiB / 16, refused, free_bytes));
        CHECK(dev.allocations == 3);
    }
    {   // more than 1 GiB where the device has it
        Device dev{170 * GiB};
        Buf b{dev, 4};
        size_t refused = ~size_t(0);
        CHECK(tmb::reserve_bitmaps(b, 5 * GiB, refused, [&] { return dev.free_bytes; }) && b.cap == 5 * GiB);
        CHECK(!tmb::reserve_bitmaps(b, 6 * GiB, refused, [&] { return dev.free_bytes; }) && b.cap == 5 * GiB);
    }
    {   // queues by their bound: refused once, then by their exact sizes
        const size_t MiB = size_t(1) << 20;
        Device dev{150 * MiB};
        Buf queue{dev, 16}, slices{dev, 4};
        size_t refused = ~size_t(0);
        for (int i = 0; i < 5; ++i) {
            CHECK(!tmb::reserve_ahead(queue, 8 * MiB, slices, 10 * MiB, 168 * MiB, 256 * MiB, refused));
            queue.reserve(MiB);
            slices.reserve(MiB);
        }
        CHECK(dev.refusals == 1);
        CHECK(tmb::reserve_ahead(queue, 4 * MiB, slices, 10 * MiB, 104 * MiB, 256 * MiB, refused));
        CHECK(!tmb::reserve_ahead(queue, 4 * MiB, slices, 10 * MiB, 104 * MiB, 100 * MiB, refused));
    }
    std::puts("ok");
}
