"""The ring that pageable inputs go through, on the CPU against a stand-in for the CUDA runtime: a stream is a thread
that runs its copies late, an event is reached when the stream has come that far, and events, page-locked memory,
threads and waits can be made to fail.  Every byte arrives whatever the chunks; what cannot be had leaves the
feed inactive with nothing held, and the next feed works; an error of a wait ends the call."""
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from native import run_native  # noqa: E402

CUDA = "/usr/local/cuda/include"

PROGRAM = r"""
#include "host_feed.h"

#include <dlfcn.h>
#include <pthread.h>

#include <atomic>
#include <cstdlib>
#include <deque>
#include <functional>

// ---- stand-in for the runtime ----
static std::mutex M;
static std::condition_variable CV;
static std::deque<std::function<void()>> work;
static bool busy = false, quit = false;
struct Event { long recorded = 0, reached = 0; };
static int fail_event_after = -1, fail_wait = 0, live_events = 0;
static std::atomic<int> fail_thread_after{-1};
static bool fail_memory = false;
static long live_blocks = 0;

static void stream_main() {
    std::unique_lock<std::mutex> g(M);
    while (true) {
        CV.wait(g, [] { return quit || !work.empty(); });
        if (work.empty()) return;
        auto op = std::move(work.front());
        work.pop_front();
        busy = true;
        g.unlock();
        if (std::rand() % 4 == 0) std::this_thread::sleep_for(std::chrono::microseconds(200));
        op();
        g.lock();
        busy = false;
        CV.notify_all();
    }
}
static void drain() {
    std::unique_lock<std::mutex> g(M);
    CV.wait(g, [] { return work.empty() && !busy; });
}
extern "C" {
cudaError_t cudaMallocHost(void** p, size_t n) {
    if (fail_memory) return cudaErrorMemoryAllocation;
    ++live_blocks;
    *p = std::malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { --live_blocks; std::free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    if (fail_event_after == 0) return cudaErrorMemoryAllocation;
    if (fail_event_after > 0) --fail_event_after;
    ++live_events;
    *e = reinterpret_cast<cudaEvent_t>(new Event());
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) { --live_events; delete reinterpret_cast<Event*>(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t ev, cudaStream_t) {
    Event* e = reinterpret_cast<Event*>(ev);
    std::lock_guard<std::mutex> g(M);
    const long at = ++e->recorded;
    work.push_back([e, at] { std::lock_guard<std::mutex> h(M); e->reached = at; });
    CV.notify_all();
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t ev) {
    Event* e = reinterpret_cast<Event*>(ev);
    if (!e) return cudaErrorInvalidResourceHandle;
    std::unique_lock<std::mutex> g(M);
    if (fail_wait > 0 && --fail_wait == 0) return cudaErrorLaunchFailure;
    const long at = e->recorded;
    CV.wait(g, [&] { return e->reached >= at; });
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::lock_guard<std::mutex> g(M);
    work.push_back([=] { std::memcpy(d, s, n); });
    CV.notify_all();
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "stand-in"; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    *a = cudaPointerAttributes{};
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
int pthread_create(pthread_t* t, const pthread_attr_t* at, void* (*f)(void*), void* arg) {
    static auto real = reinterpret_cast<int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*)>(dlsym(RTLD_NEXT, "pthread_create"));
    if (fail_thread_after == 0) return EAGAIN;
    if (fail_thread_after > 0) --fail_thread_after;
    return real(t, at, f, arg);
}
}

using namespace culsh_b200;

// source -> device in chunks, as the hashing drivers do; 1: through the ring, 0: not, -1: an error was thrown
static int send(FeedRing& ring, size_t bytes, size_t chunk, bool& same) {
    std::vector<uint8_t> src(bytes), dst(bytes, 0);
    for (size_t i = 0; i < bytes; i += 64) src[i] = (uint8_t)std::rand(), src[std::min(bytes - 1, i + 63)] = (uint8_t)(i >> 6);
    int how;
    try {
        HostFeed feed(ring, 0, nullptr, src.data(), bytes);
        how = feed.active() ? 1 : 0;
        if (how)
            for (size_t at = 0; at < bytes; at += chunk) feed.copy(dst.data() + at, at, std::min(chunk, bytes - at));
    } catch (const Error&) {
        how = -1;
    }
    drain();
    same = dst == src;
    return how;
}

#define EXPECT(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
    std::thread stream(stream_main);
    struct End { std::thread& t; ~End() { { std::lock_guard<std::mutex> g(M); quit = true; } CV.notify_all(); t.join(); } } end{stream};
    const size_t big = FEED_MIN_BYTES;
    bool same = false;
    {
        FeedRing ring;
        // no ring before the handle has been given FEED_RING_AFTER bytes, and one at once for that many
        EXPECT(send(ring, big - 1, big, same) == 0 && ring.seen == 0);
        for (size_t given = big; given < FEED_RING_AFTER; given += big)
            EXPECT(send(ring, big, big, same) == 0 && !ring.mem && live_events == 0 && live_blocks == 0);
        EXPECT(send(ring, big, big, same) == 1 && same);
        ring.release();
        EXPECT(send(ring, big, big, same) == 0);
        EXPECT(send(ring, FEED_RING_AFTER, big, same) == 1 && same);
        const size_t sizes[] = {big, big + 1, big + FEED_PIECE - 1, 3 * big + 12345, FEED_SLOTS * FEED_PIECE * 2 + big + 1};
        const size_t chunks[] = {big, FEED_PIECE, FEED_PIECE * 3 / 2 + 7, (size_t)1 << 30};
        for (size_t n : sizes)
            for (size_t c : chunks) {  // every call finds the ring as the last one left it
                EXPECT(send(ring, n, c, same) == 1);
                EXPECT(same);
            }
        // the number of events a ring needs, then one fewer
        EXPECT(live_events == FEED_SLOTS && live_blocks == 1);
        ring.release();
        EXPECT(live_events == 0 && live_blocks == 0);
        for (int n : {0, 1, FEED_SLOTS - 1}) {
            fail_event_after = n;
            ring.seen = FEED_RING_AFTER;
            EXPECT(send(ring, big, big, same) == 0);
            EXPECT(!ring.mem && live_events == 0 && live_blocks == 0);
            fail_event_after = -1;
            ring.seen = FEED_RING_AFTER;
            EXPECT(send(ring, 2 * big, big, same) == 1 && same);
            ring.release();
        }
        fail_memory = true;
        ring.seen = FEED_RING_AFTER;
        EXPECT(send(ring, big, big, same) == 0);
        EXPECT(!ring.mem && live_events == 0 && live_blocks == 0);
        fail_memory = false;
        ring.seen = FEED_RING_AFTER;
        EXPECT(send(ring, big, big, same) == 1 && same);
        // no thread, and one only
        fail_thread_after = 0;
        EXPECT(send(ring, big, big, same) == 0);
        fail_thread_after = 1;
        EXPECT(send(ring, 2 * big + 1, big, same) == 1 && same);
        fail_thread_after = -1;
        // a wait that fails ends the call, and the next one works
        fail_wait = 3;
        EXPECT(send(ring, 4 * big, big, same) == -1);
        fail_wait = 0;
        EXPECT(send(ring, 4 * big, big, same) == 1 && same);
        // a call that ends between two chunks
        {
            std::vector<uint8_t> src(4 * big, 1), dst(4 * big);
            HostFeed feed(ring, 0, nullptr, src.data(), src.size());
            feed.copy(dst.data(), 0, FEED_PIECE / 2);
            drain();
        }
        EXPECT(send(ring, 2 * big, big, same) == 1 && same);
        bool thrown = false;
        try {
            std::vector<uint8_t> src(big);
            HostFeed feed(ring, 0, nullptr, src.data(), src.size());
            feed.copy(src.data(), 1, big);
        } catch (const Error&) {
            thrown = true;
        }
        EXPECT(thrown);
        ring.release();
    }
    EXPECT(live_events == 0 && live_blocks == 0);
    std::puts("ok");
    return 0;
}
"""


@pytest.mark.skipif(not os.path.exists(os.path.join(CUDA, "cuda_runtime_api.h")), reason="no CUDA headers")
def test_ring(tmp_path):
    assert run_native(tmp_path, PROGRAM, flags=["-I", CUDA, "-ldl"], timeout=300).strip() == "ok"
