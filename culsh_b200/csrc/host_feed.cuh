// Host -> device feed of ordinary (pageable) host arrays.  A cudaMemcpyAsync from pageable memory
// goes through one driver thread that copies into a small pinned buffer: about 11 GB/s on rows a
// NumPy program holds, a fifth of what the link takes.  Here a few threads of the call copy pieces of
// the source into a ring of pinned memory kept by the handle, and the calling thread issues the
// device copies in order as the pieces become ready.
// 400,000 x 128 float32 rows (205 MB): the copies take 17.9 ms from pageable memory, 6.0 this way (34 GB/s).
#pragma once

#include <algorithm>
#include <condition_variable>
#include <mutex>
#include <thread>
#include <vector>

#include "common.cuh"

namespace culsh_b200 {

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
    HostFeed(const CtxPtr& ctx, const void* src, size_t total_bytes) : c_(ctx) {
        if (total_bytes < FEED_MIN_BYTES || !is_pageable_pointer(src)) return;
        if (!c_->feed_ring) {
            if (cudaMallocHost(&c_->feed_ring, FEED_SLOTS * FEED_PIECE) != cudaSuccess) {
                cudaGetLastError();
                c_->feed_ring = nullptr;
                return;
            }
            for (auto& e : c_->feed_free)
                if (!e) CU_CHECK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        }
        ring_ = static_cast<uint8_t*>(c_->feed_ring);
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
            CU_CHECK(cudaMemcpyAsync(out, ring_ + (piece % FEED_SLOTS) * FEED_PIECE + at, part, cudaMemcpyHostToDevice, c_->copy_stream));
            if (at + part == FEED_PIECE || begin + part == bytes_) {  // the piece has been sent whole
                CU_CHECK(cudaEventRecord(c_->feed_free[piece % FEED_SLOTS], c_->copy_stream));
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
        cudaError_t e = cudaSetDevice(c_->device);
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
            if (e == cudaSuccess) e = cudaEventSynchronize(c_->feed_free[i % FEED_SLOTS]);
            if (e == cudaSuccess)
                std::memcpy(ring_ + (i % FEED_SLOTS) * FEED_PIECE, src_ + i * FEED_PIECE, std::min(FEED_PIECE, bytes_ - i * FEED_PIECE));
            {
                std::lock_guard<std::mutex> g(m_);
                if (e != cudaSuccess) failed_ = e;
                filled_[i] = 1;
            }
            cv_.notify_all();
        }
    }

    const CtxPtr& c_;
    uint8_t* ring_ = nullptr;
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
