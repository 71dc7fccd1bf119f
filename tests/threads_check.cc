// on_threads and parallel_sort where no or few threads can be had: the address
// space is limited, so that a thread's stack is refused.
#include "../tagmatch_b200/csrc/threads.hpp"
#include <sys/resource.h>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <stdexcept>

#define CHECK(x)                                                   \
    do {                                                           \
        if (!(x)) {                                                \
            std::printf("%s:%d: %s\n", __FILE__, __LINE__, #x);    \
            std::exit(1);                                          \
        }                                                          \
    } while (0)

static void check(unsigned n) {
    std::vector<std::atomic<int>> ran(n);
    tmb::on_threads(n, [&](unsigned t) { ++ran[t]; });
    for (auto &r : ran) CHECK(r == 1);
    for (unsigned bad = 0; bad < n; bad += 1 + n / 4) {
        std::atomic<unsigned> ended{0};
        bool caught = false;
        try {
            tmb::on_threads(n, [&](unsigned t) {
                ++ended;
                if (t == bad) throw std::runtime_error("x");
            });
        } catch (const std::runtime_error &) {
            caught = true;
        }
        CHECK(caught && ended == n);
    }
}

int main() {
    std::vector<unsigned> v(300001);
    for (int limited = 0; limited < 3; ++limited) {
        if (limited) {  // no stack at all, then one or two
            long pages = 0;
            FILE *f = std::fopen("/proc/self/statm", "r");
            CHECK(f && std::fscanf(f, "%ld", &pages) == 1);
            std::fclose(f);
            const rlim_t bytes = rlim_t(pages) * 4096 + (limited == 1 ? (2u << 20) : (20u << 20));
            rlimit l{bytes, RLIM_INFINITY};
            CHECK(setrlimit(RLIMIT_AS, &l) == 0);
        }
        for (unsigned n : {0u, 1u, 2u, 3u, 32u}) check(n);
        unsigned x = 1;
        for (auto &e : v) e = x = x * 1664525u + 1013904223u;
        tmb::parallel_sort(v, [](unsigned a, unsigned b) { return a < b; });
        CHECK(std::is_sorted(v.begin(), v.end()));
    }
    std::puts("ok");
}
