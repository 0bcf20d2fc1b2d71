// Scenarios for csrc/host_staging.h on the CPU, against the stand-in runtime of fake_cuda/cuda_runtime.h.
#include "host_staging.h"

#include <cstdio>
#include <deque>
#include <new>
#include <string>

static thread_local bool t_no_memory = false;
void* operator new(size_t n) {
    void* p = t_no_memory ? nullptr : std::malloc(n);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

using namespace b200;
using Bytes = std::vector<uint8_t>;

#define CHECK(cond)                                                     \
    do {                                                                \
        if (!(cond)) {                                                  \
            std::printf("line %d: %s\n", __LINE__, #cond);              \
            return 1;                                                   \
        }                                                               \
    } while (0)

static Bytes pattern(size_t n, unsigned seed) {
    Bytes b(n);
    for (size_t i = 0; i < n; ++i) b[i] = static_cast<uint8_t>((i * 2654435761u + seed * 40503u) >> 13);
    return b;
}

// One call as the host entry makes it: up on `up`, "compute" by leaving the bytes as they are, down on `down` in slabs.
static cudaError_t call(Staging& io, fake::Stream& up, fake::Stream& down, const Bytes& in, Bytes& dev, uint8_t* out, size_t slab) {
    HostCall host(io, &up, &down);
    cudaError_t e = io.upload(dev.data(), in.data(), in.size(), &up);
    if (e != cudaSuccess) return e;
    cudaStreamSynchronize(&up);
    for (size_t at = 0; at < in.size(); at += slab) {
        const size_t n = in.size() - at < slab ? in.size() - at : slab;
        if ((e = io.download(out + at, dev.data() + at, n, &down)) != cudaSuccess) return e;
    }
    return host.finish();
}

static const size_t kSizes[] = {1, 4095, 65537, Staging::kChunk - 1, Staging::kChunk, 5 * Staging::kChunk + 13, 21 * Staging::kChunk + 1};

static int round_trip() {
    Staging io;
    fake::Stream up, down;
    for (size_t n : kSizes) {
        const Bytes in = pattern(n, 1);
        Bytes dev(n), out(n);
        CHECK(call(io, up, down, in, dev, out.data(), 3 * Staging::kChunk + 77) == cudaSuccess);
        CHECK(out == in);
    }
    io.release();
    CHECK(fake::live_events == 0 && fake::live_host == 0);
    return 0;
}

// A call that fails half way leaves nothing running: no copy is pending on a stream, the caller's memory changes no more,
// and the next call, on other streams, is correct.
static int failed_call() {
    const size_t n = 20 * Staging::kChunk + 5;
    const Bytes in = pattern(n, 2);
    for (int good : {0, 3, 21, 24, 30, 38}) {            // copies that still go out: 21 up, 21 down
        Staging io;
        fake::Stream up, down;
        Bytes dev(n), out(n);
        fake::delay_us = 3000;
        fake::fail_copy_in = good;
        CHECK(call(io, up, down, in, dev, out.data(), n) == cudaErrorInvalidValue);
        CHECK(fake::queued == 0);
        const Bytes then = out;
        std::this_thread::sleep_for(std::chrono::milliseconds(60));
        CHECK(out == then);
        fake::delay_us = 100;
        const Bytes in2 = pattern(n, 3);
        CHECK(call(io, down, up, in2, dev, out.data(), n) == cudaSuccess);
        CHECK(out == in2);
        io.release();
    }
    return 0;
}

// Where there is no pinned memory, or no event, the copies go the driver's way; nothing is lost, and a later call gets its ring.
static int no_ring() {
    const size_t n = 5 * Staging::kChunk + 13;
    const Bytes in = pattern(n, 4);
    for (int event : {-1, 0, 3, 4, 11}) {                // events that can still be made; -1: no pinned memory
        Staging io;
        fake::Stream up, down;
        Bytes dev(n), out(n), again(n);
        fake::pageable_copies_wait = true;
        for (int i = 0; i < 2; ++i) {
            (event < 0 ? fake::fail_host_alloc_in : fake::fail_event_in) = event < 0 ? 0 : event;
            Bytes got(n);
            HostCall host(io, &up, &down);
            CHECK(io.upload(dev.data(), in.data(), n, &up) == cudaSuccess);
            CHECK(fake::live_events == 0 && fake::live_host == 0);
            (event < 0 ? fake::fail_host_alloc_in : fake::fail_event_in) = event < 0 ? 0 : event;
            CHECK(io.download(got.data(), dev.data(), n, &down) == cudaSuccess);
            CHECK(fake::live_events == 0 && fake::live_host == 0);
            CHECK(host.finish() == cudaSuccess);
            CHECK(got == in);
        }
        fake::pageable_copies_wait = false;
        CHECK(call(io, up, down, in, dev, again.data(), n) == cudaSuccess);
        CHECK(again == in && fake::live_host == 1 && fake::live_events == Staging::kUp + Staging::kDown);
        io.release();
        CHECK(fake::live_events == 0 && fake::live_host == 0);
    }
    return 0;
}

// Posting copies needs no memory: the host entry is called through a C ABI, which no exception may leave.
static int no_memory() {
    const Bytes in = pattern(200 * 1024, 5);
    std::deque<CopyJob> jobs(2000);
    Bytes out(in.size() + jobs.size());
    t_no_memory = true;
    for (size_t i = 0; i < jobs.size(); ++i) CopyPool::get().post(jobs[i], out.data() + i, in.data(), i == 0 ? in.size() : 1);
    for (auto& j : jobs) CopyPool::get().wait(j);
    t_no_memory = false;
    CHECK(std::memcmp(out.data() + jobs.size(), in.data() + jobs.size(), in.size() - jobs.size()) == 0);
    return 0;
}

int main(int, char** argv) {
    const std::string what = argv[1];
    int rc = 2;
    if (what == "round_trip") rc = round_trip();
    if (what == "failed_call") rc = failed_call();
    if (what == "no_ring") rc = no_ring();
    if (what == "no_memory") rc = no_memory();
    CopyPool::get().release();
    if (rc == 0) std::printf("ok\n");
    return rc;
}
