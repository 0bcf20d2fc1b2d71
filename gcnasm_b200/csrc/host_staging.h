// Copies between pageable host memory and the GPU for b200_gemm_a8w8_host.
//
// cudaMemcpyAsync on pageable memory goes through the driver's own staging on one CPU thread: 82 MB of operands and result of a
// 4096 x 7168 x 2048 problem took 5.3 ms, 15 GB/s, against about 55 GB/s of the PCIe link in each direction.  Here the
// bytes pass through a small pinned ring, and several threads move pieces between the ring and the caller's memory while
// the copy engines work on other chunks: 2.0 ms (1.45 ms when the caller's memory is pinned and nothing is staged).
#pragma once

#include <cuda_runtime.h>
#include <emmintrin.h>
#include <sched.h>

#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace b200 {

struct CopyJob {
    uint8_t* dst = nullptr;
    const uint8_t* src = nullptr;
    size_t n = 0, taken = 0;                             // taken and next: under the pool's lock
    CopyJob* next = nullptr;
    std::atomic<size_t> left{0};
};

// Threads that work through posted copies in pieces of 64 KB.  At most eleven, started by the first large copy, asleep
// between calls (after about 100 us of spinning: the chunks of one call follow each other closely), joined by release().
// With the caller they take up three quarters of the CPUs that the process may run on: several processes of one machine
// each get their share through their affinity masks.
// Whoever waits for a job works on the queue meanwhile, so that jobs get done with no threads at all.
class CopyPool {
public:
    static CopyPool& get() {
        alignas(CopyPool) static unsigned char room[sizeof(CopyPool)];
        static CopyPool* p = new (room) CopyPool;        // never destroyed: threads may outlive static destructors
        return *p;
    }
    void post(CopyJob& j, void* dst, const void* src, size_t n) {
        j.dst = static_cast<uint8_t*>(dst);
        j.src = static_cast<const uint8_t*>(src);
        j.n = n;
        j.taken = 0;
        j.next = nullptr;
        j.left.store(n, std::memory_order_relaxed);
        if (n == 0) return;
        lock();
        (first_ ? last_->next : first_) = &j;            // (linked through the jobs: nothing here can fail)
        last_ = &j;
        queued_.fetch_add(1, std::memory_order_release);
        unlock();
        if (n < kWakeFrom) return;                       // the caller, waiting for it, does it alone
        std::lock_guard<std::mutex> lk(mu_);
        start_threads();
        if (asleep_) wake_.notify_all();
    }
    void wait(CopyJob& j) {
        while (j.left.load(std::memory_order_acquire) != 0)
            if (!step()) _mm_pause();
    }
    void release() {
        std::vector<std::thread> gone;
        {
            std::lock_guard<std::mutex> lk(mu_);
            gone.swap(threads_);
            generation_.fetch_add(1);
            wake_.notify_all();
        }
        for (auto& t : gone) t.join();
    }

private:
    static constexpr size_t kPiece = 64 * 1024, kWakeFrom = 256 * 1024;
    static constexpr unsigned kMaxThreads = 11;

    void lock() {
        while (flag_.test_and_set(std::memory_order_acquire)) _mm_pause();
    }
    void unlock() { flag_.clear(std::memory_order_release); }

    void start_threads() {
        if (!threads_.empty()) return;
        cpu_set_t set;
        unsigned cpus = 1;
        if (sched_getaffinity(0, sizeof(set), &set) == 0) cpus = static_cast<unsigned>(CPU_COUNT(&set));
        unsigned want = cpus * 3 / 4;                    // the caller is one of them
        want = want > kMaxThreads + 1 ? kMaxThreads : (want ? want - 1 : 0);
        const unsigned g = generation_.load();
        for (unsigned i = 0; i < want; ++i) {
            try {
                threads_.emplace_back([this, g] { loop(g); });
            } catch (...) {
                break;
            }
        }
    }
    void loop(unsigned g) {
        while (generation_.load(std::memory_order_relaxed) == g) {
            if (step()) continue;
            for (int i = 0; i < 2000 && queued_.load(std::memory_order_acquire) == 0; ++i) _mm_pause();
            if (queued_.load(std::memory_order_acquire) != 0) continue;
            std::unique_lock<std::mutex> lk(mu_);
            ++asleep_;
            wake_.wait(lk, [&] { return queued_.load(std::memory_order_acquire) != 0 || generation_.load() != g; });
            --asleep_;
        }
    }
    // takes and copies one piece of the oldest job; false when the queue is empty
    bool step() {
        if (queued_.load(std::memory_order_acquire) == 0) return false;
        lock();
        CopyJob* j = first_;
        if (!j) {
            unlock();
            return false;
        }
        const size_t at = j->taken, c = j->n - at < kPiece ? j->n - at : kPiece;
        j->taken += c;
        if (j->taken == j->n) {
            first_ = j->next;
            queued_.fetch_sub(1, std::memory_order_relaxed);
        }
        unlock();
        piece(j->dst + at, j->src + at, c);
        j->left.fetch_sub(c, std::memory_order_release);
        return true;
    }
    // Neither side is in this core's caches (a DMA has written one, the caller owns the other): non-temporal stores spare the
    // read of the destination, and the prefetch carries on over the 4 KB boundaries where the hardware's stops.  From and
    // to DRAM: memcpy 48 GB/s on 8 threads and 58 on 12, this 73 and 80.
    static void piece(uint8_t* d, const uint8_t* s, size_t n) {
        if (n >= 4096) {
            const size_t head = (16 - (reinterpret_cast<uintptr_t>(d) & 15)) & 15;
            std::memcpy(d, s, head);
            d += head;
            s += head;
            n -= head;
            for (; n >= 64; n -= 64, d += 64, s += 64) {
                _mm_prefetch(reinterpret_cast<const char*>(s) + 2048, _MM_HINT_T0);
                __m128i v[4];
                for (int i = 0; i < 4; ++i) v[i] = _mm_loadu_si128(reinterpret_cast<const __m128i*>(s) + i);
                for (int i = 0; i < 4; ++i) _mm_stream_si128(reinterpret_cast<__m128i*>(d) + i, v[i]);
            }
            _mm_sfence();
        }
        std::memcpy(d, s, n);
    }

    std::atomic_flag flag_ = ATOMIC_FLAG_INIT;           // guards the queue and the jobs' `taken`
    CopyJob *first_ = nullptr, *last_ = nullptr;         // the queue, oldest first
    std::atomic<unsigned> queued_{0}, generation_{0};
    std::mutex mu_;                                      // guards threads_ and asleep_
    std::condition_variable wake_;
    std::vector<std::thread> threads_;
    int asleep_ = 0;
};

// The pinned ring of one device and the copies of one call through it.  Upload chunks and result chunks have their own slots.
// 2 MB chunks: about 40 us of PCIe time each, so that the last chunk's host copy, which nothing hides, stays short.
class Staging {
public:
    static constexpr size_t kChunk = size_t(2) << 20;
    static constexpr int kUp = 4, kDown = 8;

    static bool pageable(const void* p) {
        cudaPointerAttributes a;
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
            cudaGetLastError();
            return true;
        }
        return a.type == cudaMemoryTypeUnregistered;
    }
    // Queued on `st`; the caller's memory has been read when this returns, or (pinned memory) when the stream gets there.
    cudaError_t upload(void* dev, const void* host, size_t n, cudaStream_t st) {
        if (!pageable(host) || !prepare()) return cudaMemcpyAsync(dev, host, n, cudaMemcpyHostToDevice, st);
        cudaError_t e = cudaSuccess;
        const size_t chunks = (n + kChunk - 1) / kChunk;
        const unsigned first = up_next_;
        auto bytes = [&](size_t i) { return n - i * kChunk < kChunk ? n - i * kChunk : kChunk; };
        // chunk i is copied by the pool while chunk i - 1 waits for its copy and goes to the copy engine
        for (size_t i = 0; i <= chunks && e == cudaSuccess; ++i) {
            if (i < chunks) {
                const int slot = up_next_++ % kUp;
                if ((e = cudaEventSynchronize(up_free_[slot])) != cudaSuccess) break;
                CopyPool::get().post(up_job_[slot], ring_ + slot * kChunk, static_cast<const uint8_t*>(host) + i * kChunk, bytes(i));
            }
            if (i > 0) {
                const int slot = (first + i - 1) % kUp;
                if ((e = post_arrived()) != cudaSuccess) break;
                CopyPool::get().wait(up_job_[slot]);
                e = cudaMemcpyAsync(static_cast<uint8_t*>(dev) + (i - 1) * kChunk, ring_ + slot * kChunk, bytes(i - 1), cudaMemcpyHostToDevice, st);
                if (e == cudaSuccess) e = cudaEventRecord(up_free_[slot], st);
            }
        }
        for (auto& j : up_job_) CopyPool::get().wait(j);
        return e;
    }
    // Queued on `st`; what goes through the ring is in the caller's memory after finish_downloads().
    cudaError_t download(void* host, const void* dev, size_t n, cudaStream_t st) {
        if (!pageable(host) || !prepare()) return cudaMemcpyAsync(host, dev, n, cudaMemcpyDeviceToHost, st);
        cudaError_t e = cudaSuccess;
        for (size_t at = 0; at < n && e == cudaSuccess; at += kChunk) {
            const size_t c = n - at < kChunk ? n - at : kChunk;
            const int slot = issued_ % kDown;
            if ((e = post_arrived()) != cudaSuccess) break;
            if (issued_ - posted_ == kDown && (e = post_oldest()) != cudaSuccess) break;
            CopyPool::get().wait(down_job_[slot]);                   // the chunk that had the slot before
            e = cudaMemcpyAsync(ring_ + (kUp + slot) * kChunk, static_cast<const uint8_t*>(dev) + at, c, cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaEventRecord(down_done_[slot], st);
            if (e != cudaSuccess) break;
            down_to_[slot] = static_cast<uint8_t*>(host) + at;
            down_bytes_[slot] = c;
            ++issued_;
        }
        return e;
    }
    cudaError_t finish_downloads() {
        cudaError_t e = cudaSuccess;
        while (posted_ != issued_ && e == cudaSuccess) e = post_oldest();
        for (auto& j : down_job_) CopyPool::get().wait(j);
        return e;
    }
    // The end of a call that failed half way: waits for what its streams hold (copies into the ring and into pinned memory)
    // and for the pieces that copy threads still move, so that nothing touches the caller's memory or the ring any
    // more.  Results that only reached the ring are dropped.
    void settle(cudaStream_t st, cudaStream_t copies) {
        cudaStreamSynchronize(st);
        if (copies) cudaStreamSynchronize(copies);
        cudaGetLastError();
        for (auto& j : up_job_) CopyPool::get().wait(j);
        for (auto& j : down_job_) CopyPool::get().wait(j);
        posted_ = issued_ = 0;
    }
    void release() {
        auto destroy = [](cudaEvent_t& e) {
            if (e) cudaEventDestroy(e);
            e = nullptr;
        };
        for (auto& e : up_free_) destroy(e);
        for (auto& e : down_done_) destroy(e);
        if (ring_) cudaFreeHost(ring_);
        ring_ = nullptr;
    }

private:
    // False where there is no pinned memory to be had (a process near its limit on locked memory): the driver then stages
    // the copies, slower, and the next call asks again.
    bool prepare() {
        if (ring_) return true;
        void* p = nullptr;
        cudaError_t e = cudaHostAlloc(&p, (kUp + kDown) * kChunk, cudaHostAllocDefault);
        if (e == cudaSuccess) ring_ = static_cast<uint8_t*>(p);
        for (int i = 0; i < kUp && e == cudaSuccess; ++i) e = cudaEventCreateWithFlags(&up_free_[i], cudaEventDisableTiming);
        for (int i = 0; i < kDown && e == cudaSuccess; ++i) e = cudaEventCreateWithFlags(&down_done_[i], cudaEventDisableTiming);
        if (e == cudaSuccess) return true;
        cudaGetLastError();
        release();
        return false;
    }
    // result chunks that have arrived in the ring go to the pool
    cudaError_t post_arrived() {
        while (posted_ != issued_) {
            const cudaError_t e = cudaEventQuery(down_done_[posted_ % kDown]);
            if (e == cudaErrorNotReady) {
                cudaGetLastError();
                return cudaSuccess;
            }
            if (e != cudaSuccess) return e;
            post_next();
        }
        return cudaSuccess;
    }
    cudaError_t post_oldest() {
        const cudaError_t e = cudaEventSynchronize(down_done_[posted_ % kDown]);
        if (e == cudaSuccess) post_next();
        return e;
    }
    void post_next() {
        const int slot = posted_++ % kDown;
        CopyPool::get().post(down_job_[slot], down_to_[slot], ring_ + (kUp + slot) * kChunk, down_bytes_[slot]);
    }

    uint8_t* ring_ = nullptr;
    cudaEvent_t up_free_[kUp] = {}, down_done_[kDown] = {};
    CopyJob up_job_[kUp], down_job_[kDown];
    unsigned up_next_ = 0, issued_ = 0, posted_ = 0;     // chunks: of all uploads; results whose DMA is queued; ... handed to the pool
    uint8_t* down_to_[kDown] = {};
    size_t down_bytes_[kDown] = {};
};

// One call through the ring, on stream `st` and, for results, `copies` (or null).  Whichever way the call ends, nothing of it
// is left running: finish() on the way that succeeds, the destructor on every other one.
class HostCall {
public:
    HostCall(Staging& io, cudaStream_t st, cudaStream_t copies) : io_(io), st_(st), copies_(copies) {}
    HostCall(const HostCall&) = delete;
    ~HostCall() {
        if (!finished_) io_.settle(st_, copies_);
    }
    // The results are in the caller's memory and `st`, which waits for `copies`, is idle.
    cudaError_t finish() {
        cudaError_t e = io_.finish_downloads();
        if (e == cudaSuccess) e = cudaStreamSynchronize(st_);
        finished_ = e == cudaSuccess;
        return e;
    }

private:
    Staging& io_;
    cudaStream_t st_, copies_;
    bool finished_ = false;
};

}  // namespace b200
