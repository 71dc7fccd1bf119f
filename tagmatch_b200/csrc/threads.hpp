// Host work spread over threads.
#pragma once
#include <algorithm>
#include <cstddef>
#include <exception>
#include <thread>
#include <vector>

namespace tmb {

inline unsigned worker_threads() { return std::max(1u, std::min(32u, std::thread::hardware_concurrency())); }

// Runs f(0) .. f(n - 1), each on a thread of its own but the first, which is
// the caller's, as are those that no thread can be had for.  An exception of
// f (memory) is thrown again here, once all have ended.
template <class F>
void on_threads(unsigned n, F f) {
    std::vector<std::exception_ptr> failed(n);
    auto run = [&](unsigned t) {
        try {
            f(t);
        } catch (...) {
            failed[t] = std::current_exception();
        }
    };
    std::vector<std::thread> ts;
    ts.reserve(n);
    unsigned next = 1;
    try {
        for (; next < n; ++next) ts.emplace_back(run, next);
    } catch (...) {  // no thread, or no memory for one: [next, n) are left
    }
    if (n) run(0);
    for (; next < n; ++next) run(next);
    for (auto &x : ts) x.join();
    for (auto &e : failed)
        if (e) std::rethrow_exception(e);
}

// Sorts v with cmp on all hardware threads: sorted chunks, then pairwise
// merges.
template <class T, class Cmp>
void parallel_sort(std::vector<T> &v, Cmp cmp) {
    const size_t n = v.size();
    const unsigned th = worker_threads();
    if (n < (size_t(1) << 16) || th == 1) {
        std::sort(v.begin(), v.end(), cmp);
        return;
    }
    std::vector<size_t> b(th + 1);
    for (unsigned i = 0; i <= th; ++i) b[i] = n * i / th;
    on_threads(th, [&](unsigned i) { std::sort(v.begin() + b[i], v.begin() + b[i + 1], cmp); });
    for (unsigned w = 1; w < th; w *= 2)
        on_threads((th - w + 2 * w - 1) / (2 * w), [&](unsigned k) {
            const unsigned i = 2 * w * k;
            std::inplace_merge(v.begin() + b[i], v.begin() + b[i + w], v.begin() + b[std::min(i + 2 * w, th)], cmp);
        });
}

}  // namespace tmb
