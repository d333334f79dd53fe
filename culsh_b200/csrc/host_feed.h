// Host -> device feed of ordinary (pageable) host arrays.  A cudaMemcpyAsync from pageable memory
// goes through one driver thread that copies into a small pinned buffer: about 11 GB/s on rows a
// NumPy program holds, a fifth of what the link takes.  Here a few threads of the call copy pieces of
// the source into a ring of pinned memory kept by the handle, and the calling thread issues the
// device copies in order as the pieces become ready.
// 400,000 x 128 float32 rows (205 MB): the copies take 17.9 ms from pageable memory, 6.0 this way (34 GB/s).
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

constexpr int FEED_SLOTS = 16;
constexpr size_t FEED_PIECE = (size_t)2 << 20;

// The pinned ring of a handle.
struct FeedRing {
    uint8_t* mem = nullptr;                // FEED_SLOTS pieces
    cudaEvent_t sent[FEED_SLOTS] = {};     // the last copy out of a slot

    // False, and nothing is held, when the memory or an event cannot be had.
    bool make() {
        if (mem) return true;
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

// Below this the driver's own staging is over before the threads are up.
constexpr size_t FEED_MIN_BYTES = (size_t)8 << 20;
constexpr int FEED_MAX_THREADS = 8;

class HostFeed {
public:
    // Nothing runs (active() is false) when the source is small or not pageable, when the pinned ring
    // cannot be had or no thread starts: the caller copies straight from the source then.
    HostFeed(FeedRing& ring, int device, cudaStream_t copy_stream, const void* src, size_t total_bytes)
        : ring_(ring), device_(device), stream_(copy_stream) {
        if (total_bytes < FEED_MIN_BYTES || !is_pageable_pointer(src) || !ring_.make()) return;
        src_ = static_cast<const uint8_t*>(src);
        bytes_ = total_bytes;
        n_ = ceil_div(total_bytes, FEED_PIECE);
        filled_.assign(n_, 0);
        const unsigned cores = std::max(1u, std::thread::hardware_concurrency());
        const size_t want = std::min<size_t>({(size_t)FEED_MAX_THREADS, (size_t)std::max(1u, cores - 1), n_});
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
