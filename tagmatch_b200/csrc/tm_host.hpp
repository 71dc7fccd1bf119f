// Host-side helpers: CUDA error handling and grow-only device buffers.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <algorithm>
#include <cstdio>
#include <stdexcept>
#include <string>
#include <utility>
#include <vector>

namespace tmb {

// Raised inside the engine; the C ABI turns it into a status code and a
// message (tm_last_error), so no CUDA failure ends the process.
struct Error : std::runtime_error {
    int status;
    Error(int st, const std::string &msg) : std::runtime_error(msg), status(st) {}
};

inline std::string cuda_msg(cudaError_t e, const char *what, const char *file, int line) {
    char buf[512];
    std::snprintf(buf, sizeof(buf), "%s: %s (%s:%d)", what, cudaGetErrorString(e), file, line);
    return buf;
}

#define TM_CUDA(x)                                                                       \
    do {                                                                                 \
        cudaError_t e_ = (x);                                                            \
        if (e_ != cudaSuccess) throw ::tmb::Error(-2, ::tmb::cuda_msg(e_, #x, __FILE__, __LINE__)); \
    } while (0)

#define TM_CHECK_LAUNCH() TM_CUDA(cudaGetLastError())

// Grow-only device buffer.  reserve() keeps the old contents only when it
// does not reallocate; callers treat a grown buffer as uninitialised.
template <class T>
struct DevBuf {
    T *p = nullptr;
    size_t cap = 0;
    bool owned = true;  // false: part of another allocation (borrow)
    DevBuf() = default;
    DevBuf(const DevBuf &) = delete;
    DevBuf &operator=(const DevBuf &) = delete;
    DevBuf(DevBuf &&o) noexcept : p(o.p), cap(o.cap), owned(o.owned) { o.forget(); }
    DevBuf &operator=(DevBuf &&o) noexcept {
        if (this != &o) {
            release();
            p = o.p;
            cap = o.cap;
            owned = o.owned;
            o.forget();
        }
        return *this;
    }
    ~DevBuf() { release(); }
    // Starts on n elements at q, which the caller keeps alive; growing past
    // them takes an allocation of its own.
    void borrow(T *q, size_t n) {
        release();
        p = q;
        cap = n;
        owned = false;
    }
    void forget() {
        p = nullptr;
        cap = 0;
        owned = true;
    }
    // Grows by at least half the current capacity, so a slowly growing
    // demand reallocates (and frees, which synchronises the device) rarely.
    void reserve(size_t n) {
        size_t bytes = 0;
        const cudaError_t e = grow(n, bytes);
        if (e != cudaSuccess)
            throw Error(-5, cuda_msg(e, "cudaMalloc", __FILE__, __LINE__) + " bytes=" + std::to_string(bytes));
    }
    // reserve() that reports a refusal, which leaves the buffer empty.
    bool try_reserve(size_t n) {
        size_t bytes = 0;
        return grow(n, bytes) == cudaSuccess;
    }
    void release() {
        if (p && owned) cudaFree(p);
        forget();
    }
    T *get() const { return p; }

private:
    cudaError_t grow(size_t n, size_t &bytes) {
        if (n <= cap && p) return cudaSuccess;
        if (p) n = std::max(n, cap + cap / 2);
        release();
        bytes = (n ? n : 1) * sizeof(T);
        const cudaError_t e = cudaMalloc(&p, bytes);
        if (e != cudaSuccess) {
            forget();
            cudaGetLastError();
            return e;
        }
        cap = n ? n : 1;
        return e;
    }
};

// One device allocation cut into 256-byte aligned pieces, for calls that need
// many buffers at once (an allocation and its release take 0.1-0.3 ms each).
// want() states the pieces, then allocate() hands them out.
class DevPieces {
public:
    template <class T>
    void want(DevBuf<T> &b, size_t n) {
        const size_t count = n ? n : 1;
        pieces_.push_back(Piece{&b, total_, count, [](void *buf, unsigned char *at, size_t elements) {
                                    static_cast<DevBuf<T> *>(buf)->borrow(reinterpret_cast<T *>(at), elements);
                                }});
        total_ = (total_ + count * sizeof(T) + 255) & ~size_t(255);
    }
    // block must outlive the buffers
    void allocate(DevBuf<unsigned char> &block) {
        block.reserve(total_);
        for (const Piece &x : pieces_) x.hand(x.buf, block.p + x.at, x.count);
        pieces_.clear();
        total_ = 0;
    }

private:
    struct Piece {
        void *buf;
        size_t at, count;
        void (*hand)(void *, unsigned char *, size_t);
    };
    size_t total_ = 0;
    std::vector<Piece> pieces_;
};

// A stream for work beside the owner's: fork() makes it wait for what st holds
// so far and returns it, join() makes st wait for it.  Created at first use
// on the then current device.
struct SideStream {
    cudaStream_t stream = nullptr;
    cudaEvent_t forked = nullptr, joined = nullptr;
    SideStream() = default;
    SideStream(const SideStream &) = delete;
    SideStream &operator=(const SideStream &) = delete;
    ~SideStream() { release(); }
    void release() {
        if (stream) cudaStreamDestroy(stream);
        if (forked) cudaEventDestroy(forked);
        if (joined) cudaEventDestroy(joined);
        stream = nullptr;
        forked = joined = nullptr;
    }
    void swap(SideStream &o) {
        std::swap(stream, o.stream);
        std::swap(forked, o.forked);
        std::swap(joined, o.joined);
    }
    cudaStream_t fork(cudaStream_t st) {
        if (!stream) TM_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
        if (!forked) TM_CUDA(cudaEventCreateWithFlags(&forked, cudaEventDisableTiming));
        if (!joined) TM_CUDA(cudaEventCreateWithFlags(&joined, cudaEventDisableTiming));
        TM_CUDA(cudaEventRecord(forked, st));
        TM_CUDA(cudaStreamWaitEvent(stream, forked, 0));
        return stream;
    }
    void join(cudaStream_t st) {
        TM_CUDA(cudaEventRecord(joined, stream));
        TM_CUDA(cudaStreamWaitEvent(st, joined, 0));
    }
};

// Pinned host buffer (grow-only).
template <class T>
struct HostBuf {
    T *p = nullptr;
    size_t cap = 0;
    HostBuf() = default;
    HostBuf(const HostBuf &) = delete;
    HostBuf &operator=(const HostBuf &) = delete;
    HostBuf(HostBuf &&o) noexcept : p(o.p), cap(o.cap) { o.p = nullptr; o.cap = 0; }
    ~HostBuf() { release(); }
    void reserve(size_t n) {
        if (n <= cap && p) return;
        if (p) n = std::max(n, cap + cap / 2);
        release();
        size_t bytes = (n ? n : 1) * sizeof(T);
        cudaError_t e = cudaMallocHost(&p, bytes);
        if (e != cudaSuccess) {
            p = nullptr;
            cap = 0;
            cudaGetLastError();
            throw Error(-5, cuda_msg(e, "cudaMallocHost", __FILE__, __LINE__));
        }
        cap = n ? n : 1;
    }
    void release() {
        if (p) cudaFreeHost(p);
        p = nullptr;
        cap = 0;
    }
};

// Pinned host buffer mapped into the device address space (grow-only).
// Kernels store small results into it (d); the host reads them (h) after a
// stream synchronisation.  Such stores leave the SMs over PCIe directly, so
// unlike a cudaMemcpyAsync they do not queue on a copy engine behind large
// copies that other streams have issued.
template <class T>
struct MappedBuf {
    T *h = nullptr;
    T *d = nullptr;
    size_t cap = 0;
    MappedBuf() = default;
    MappedBuf(const MappedBuf &) = delete;
    MappedBuf &operator=(const MappedBuf &) = delete;
    MappedBuf(MappedBuf &&o) noexcept : h(o.h), d(o.d), cap(o.cap) {
        o.h = o.d = nullptr;
        o.cap = 0;
    }
    MappedBuf &operator=(MappedBuf &&o) noexcept {
        if (this != &o) {
            release();
            h = o.h;
            d = o.d;
            cap = o.cap;
            o.h = o.d = nullptr;
            o.cap = 0;
        }
        return *this;
    }
    ~MappedBuf() { release(); }
    void reserve(size_t n) {
        if (n <= cap && h) return;
        if (h) n = std::max(n, cap + cap / 2);
        release();
        const size_t bytes = (n ? n : 1) * sizeof(T);
        cudaError_t e = cudaHostAlloc(reinterpret_cast<void **>(&h), bytes, cudaHostAllocMapped);
        if (e == cudaSuccess) e = cudaHostGetDevicePointer(reinterpret_cast<void **>(&d), h, 0);
        if (e != cudaSuccess) {
            if (h) cudaFreeHost(h);
            h = d = nullptr;
            cap = 0;
            cudaGetLastError();
            throw Error(-5, cuda_msg(e, "cudaHostAlloc(mapped)", __FILE__, __LINE__));
        }
        cap = n ? n : 1;
    }
    void release() {
        if (h) cudaFreeHost(h);
        h = d = nullptr;
        cap = 0;
    }
};

}  // namespace tmb
