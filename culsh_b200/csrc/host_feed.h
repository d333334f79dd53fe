// Host -> device feed of ordinary (pageable) host arrays.  A cudaMemcpyAsync from pageable memory
// goes through one driver thread that copies into a small pinned buffer: about 11 GB/s on rows a
// NumPy program holds, a fifth of what the link takes.  Here a few threads of the call copy pieces of
// the source into a ring of pinned memory kept by the handle, and the calling thread issues the
// device copies in order as the pieces become ready.
// A fit of 256 MB of float32 rows: 23.6 ms from pageable memory, 6.7 this way; 64 MB: 4.0 and 2.1.
#pragma once

#include <algorithm>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "check.h"

namespace culsh_b200 {

// 8 pieces of 2 MB.  A ring of 16 and 8 threads were no faster for 256 MB and more (6.9 ms against 6.6 - 6.8, 1 GB
// 22.9 against 23.2), slower for less (32 MB 2.0 against 1.4, 64 MB 2.7 against 2.1), and 32 MB take twice
// as long to page-lock.
constexpr int FEED_SLOTS = 8;
constexpr size_t FEED_PIECE = (size_t)2 << 20;
// Four threads read as fast as the link takes it until the source is far beyond the caches (1 GB: 24.6 ms with
// four, 23.2 with six; 64 MB: 2.1 and 2.5).
inline size_t feed_threads(size_t bytes) { return bytes < ((size_t)256 << 20) ? 4 : 6; }
// Below this the driver's own staging is as fast, because the threads have to start (16 MB: 0.94 ms direct, 1.1
// through the ring; 24 MB: 1.35 and 1.3; 32 MB: 1.74 and 1.4).
constexpr size_t FEED_MIN_BYTES = (size_t)32 << 20;
// The ring takes about 10 ms to make, what 160 MB gain by it: a handle makes it when it has been given so
// much, so that a program of one or two small fits does not pay for it.
constexpr size_t FEED_RING_AFTER = (size_t)160 << 20;

// The pinned ring of a handle.
struct FeedRing {
    uint8_t* mem = nullptr;                // FEED_SLOTS pieces
    size_t seen = 0;                       // bytes of sources that could have used it
    cudaEvent_t sent[FEED_SLOTS] = {};     // the last copy out of a slot

    // False, and nothing is held, before the handle has been given FEED_RING_AFTER bytes, these included,
    // or when the memory or an event cannot be had.
    bool make(size_t bytes) {
        if (mem) return true;
        seen += std::min(bytes, FEED_RING_AFTER);
        if (seen < FEED_RING_AFTER) return false;
        bool ok = true;
        for (auto& e : sent) {
            if (ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
                e = nullptr;
                ok = false;
            }
        }
        void* p = nullptr;
        ok = ok && cudaMallocHost(&p, FEED_SLOTS * FEED_PIECE) == cudaSuccess;
        if (ok) {
            mem = static_cast<uint8_t*>(p);
        } else {
            cudaGetLastError();
            release();
        }
        return ok;
    }
    void release() {
        for (auto& e : sent) {
            if (e) cudaEventDestroy(e);
            e = nullptr;
        }
        if (mem) cudaFreeHost(mem);
        mem = nullptr;
        seen = 0;
    }
};

// True for memory the driver does not know: a copy from it is staged.
inline bool is_pageable_pointer(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

class HostFeed {
public:
    // Nothing runs (active() is false) when the source is small or not pageable, when there is no pinned ring
    // yet or it cannot be had, or when no thread starts: the caller copies straight from the source then.
    HostFeed(FeedRing& ring, int device, cudaStream_t copy_stream, const void* src, size_t total_bytes)
        : ring_(ring), device_(device), stream_(copy_stream) {
        if (total_bytes < FEED_MIN_BYTES || !is_pageable_pointer(src) || !ring_.make(total_bytes)) return;
        src_ = static_cast<const uint8_t*>(src);
        bytes_ = total_bytes;
        n_ = ceil_div(total_bytes, FEED_PIECE);
        filled_.assign(n_, 0);
        const unsigned cores = std::max(1u, std::thread::hardware_concurrency());
        const size_t want = std::min<size_t>({feed_threads(total_bytes), (size_t)std::max(1u, cores - 1), n_});
        workers_.reserve(want);
        try {
            for (size_t i = 0; i < want; ++i) workers_.emplace_back([this] { work(); });
        } catch (...) {  // fewer threads than asked for; those that run have to be joined
        }
    }
    HostFeed(const HostFeed&) = delete;
    HostFeed& operator=(const HostFeed&) = delete;
    ~HostFeed() {
        {
            std::lock_guard<std::mutex> g(m_);
            stop_ = true;
        }
        cv_.notify_all();
        for (auto& t : workers_) t.join();
    }
    bool active() const { return !workers_.empty(); }

    // Queue on the copy stream: source bytes [begin, begin + bytes) to dst.  The ranges of successive
    // calls have to follow one another.
    void copy(void* dst, size_t begin, size_t bytes) {
        if (begin + bytes > bytes_) fail(CULSH_ERR_INVALID, "host feed: range outside of the source");
        uint8_t* out = static_cast<uint8_t*>(dst);
        while (bytes) {
            const size_t piece = begin / FEED_PIECE, at = begin % FEED_PIECE;
            const size_t part = std::min(bytes, FEED_PIECE - at);
            {
                std::unique_lock<std::mutex> g(m_);
                cv_.wait(g, [&] { return filled_[piece] != 0; });
                if (failed_ != cudaSuccess) fail(CULSH_ERR_CUDA, "host feed: %s", cudaGetErrorString(failed_));
            }
            CU_CHECK(cudaMemcpyAsync(out, ring_.mem + (piece % FEED_SLOTS) * FEED_PIECE + at, part, cudaMemcpyHostToDevice, stream_));
            if (at + part == FEED_PIECE || begin + part == bytes_) {  // the piece has been sent whole
                CU_CHECK(cudaEventRecord(ring_.sent[piece % FEED_SLOTS], stream_));
                {
                    std::lock_guard<std::mutex> g(m_);
                    sent_ = piece + 1;
                }
                cv_.notify_all();
            }
            out += part;
            begin += part;
            bytes -= part;
        }
    }

private:
    void work() {
        cudaError_t e = cudaSetDevice(device_);
        while (true) {
            size_t i;
            {
                std::unique_lock<std::mutex> g(m_);
                if (next_ >= n_ || stop_) return;
                i = next_++;
                cv_.wait(g, [&] { return stop_ || i < sent_ + FEED_SLOTS; });  // the slot's last piece is queued ...
                if (stop_) return;
            }
            // ... and has left it (a piece of an earlier call may still be on its way, too)
            if (e == cudaSuccess) e = cudaEventSynchronize(ring_.sent[i % FEED_SLOTS]);
            if (e == cudaSuccess)
                std::memcpy(ring_.mem + (i % FEED_SLOTS) * FEED_PIECE, src_ + i * FEED_PIECE, std::min(FEED_PIECE, bytes_ - i * FEED_PIECE));
            {
                std::lock_guard<std::mutex> g(m_);
                if (e != cudaSuccess) failed_ = e;
                filled_[i] = 1;
            }
            cv_.notify_all();
        }
    }

    FeedRing& ring_;
    const int device_;
    const cudaStream_t stream_;
    const uint8_t* src_ = nullptr;
    size_t bytes_ = 0, n_ = 0;
    std::mutex m_;
    std::condition_variable cv_;
    std::vector<char> filled_;
    size_t next_ = 0, sent_ = 0;
    bool stop_ = false;
    cudaError_t failed_ = cudaSuccess;
    std::vector<std::thread> workers_;
};

}  // namespace culsh_b200
