// The few runtime calls that csrc/host_staging.h makes, on the CPU: a stream is a thread that works through its queue some time
// later, device memory is host memory, and single calls can be made to fail.
#pragma once

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <mutex>
#include <thread>

enum cudaError_t { cudaSuccess = 0, cudaErrorInvalidValue = 1, cudaErrorMemoryAllocation = 2, cudaErrorNotReady = 600 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2 };
enum cudaMemoryType { cudaMemoryTypeUnregistered = 0, cudaMemoryTypeHost = 1 };
enum { cudaHostAllocDefault = 0, cudaEventDisableTiming = 2 };
struct cudaPointerAttributes { cudaMemoryType type; };

namespace fake {
inline std::atomic<int> fail_copy_in{-1}, fail_event_in{-1}, fail_host_alloc_in{-1};       // calls that still succeed; -1: all
inline std::atomic<int> live_events{0}, live_host{0}, queued{0};
inline std::atomic<int> delay_us{200};                                                       // of every copy
inline std::atomic<bool> pageable_copies_wait{false};                                        // a copy is complete when its call returns
inline bool fails(std::atomic<int>& left) { return left.load() >= 0 && left.fetch_sub(1) == 0; }

struct Stream {
    std::mutex mu;
    std::condition_variable cv;
    std::deque<std::function<void()>> q;
    bool busy = false, stop = false;
    std::thread t{[this] { run(); }};
    void run() {
        std::unique_lock<std::mutex> lk(mu);
        for (;;) {
            cv.wait(lk, [&] { return stop || !q.empty(); });
            if (q.empty()) return;
            auto f = std::move(q.front());
            q.pop_front();
            busy = true;
            lk.unlock();
            f();
            --queued;
            lk.lock();
            busy = false;
            cv.notify_all();
        }
    }
    void push(std::function<void()> f) {
        ++queued;
        std::lock_guard<std::mutex> lk(mu);
        q.push_back(std::move(f));
        cv.notify_all();
    }
    void drain() {
        std::unique_lock<std::mutex> lk(mu);
        cv.wait(lk, [&] { return q.empty() && !busy; });
    }
    ~Stream() {
        {
            std::lock_guard<std::mutex> lk(mu);
            stop = true;
            cv.notify_all();
        }
        t.join();
    }
};
struct Event { std::atomic<long> recorded{0}, done{0}; };
}  // namespace fake

using cudaStream_t = fake::Stream*;
using cudaEvent_t = fake::Event*;

inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
inline cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    if (fake::fails(fake::fail_host_alloc_in)) return cudaErrorMemoryAllocation;
    ++fake::live_host;
    *p = std::malloc(n);
    return cudaSuccess;
}
inline cudaError_t cudaFreeHost(void* p) {
    --fake::live_host;
    std::free(p);
    return cudaSuccess;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    if (fake::fails(fake::fail_event_in)) return cudaErrorMemoryAllocation;
    ++fake::live_events;
    *e = new fake::Event;
    return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e) {
    if (!e) return cudaErrorInvalidValue;
    --fake::live_events;
    delete e;
    return cudaSuccess;
}
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    const long n = ++e->recorded;
    s->push([e, n] { e->done = n; });
    return cudaSuccess;
}
inline cudaError_t cudaEventQuery(cudaEvent_t e) { return e->done >= e->recorded ? cudaSuccess : cudaErrorNotReady; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    while (cudaEventQuery(e) != cudaSuccess) std::this_thread::yield();
    return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    s->drain();
    return cudaSuccess;
}
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    if (fake::fails(fake::fail_copy_in)) return cudaErrorInvalidValue;
    st->push([=] {
        std::this_thread::sleep_for(std::chrono::microseconds(fake::delay_us.load()));
        std::memcpy(d, s, n);
    });
    if (fake::pageable_copies_wait) st->drain();
    return cudaSuccess;
}
