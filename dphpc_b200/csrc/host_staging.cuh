// Host <-> device copies of PAGEABLE host memory (the std::vector containers of the reference's harness).
//
// The driver stages such a copy through its own pinned buffer on one thread, which on this class of host moves about
// 10 GB/s -- a fifth of what the link carries from pinned memory.  Here the staging is done by a small pool of host
// threads: a copy is cut into 4 MiB pieces, the pool memcpy()s piece c+1 into one of three pinned ring buffers while the DMA
// engine moves piece c, and the other way round for downloads.  Pinned or registered host memory and device memory take
// the direct cudaMemcpyAsync path.  Like a pageable cudaMemcpyAsync, a staged call returns when the caller's buffer is
// free again (uploads) or filled (downloads).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdlib>
#include <cstdint>
#include <cstring>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

namespace sddmm {

// A fixed pool of host threads that runs "slice k of n" jobs; the caller takes part.  A staged copy hands over a piece every
// hundred microseconds, so the threads look for the next job for a while before they go to sleep, and a slice is taken
// with one compare-and-swap on {job, slices, next slice}.
class HostPool {
public:
    static HostPool &instance() {
        static HostPool pool;
        return pool;
    }
    int width() const { return static_cast<int>(workers_.size()) + 1; }
    // fn(k) for k in [0, n), spread over the pool; returns when all are done
    void run(int n, const std::function<void(int)> &fn) {
        if (n <= 1 || n > kMaxSlices || workers_.empty()) {
            for (int k = 0; k < n; ++k) fn(k);
            return;
        }
        std::lock_guard<std::mutex> one_at_a_time(run_mu_);   // callers on different host threads (one per device) take turns
        job_ = &fn;                                           // (nobody holds a slice of the previous job any more: pending_ was 0)
        pending_.store(n, std::memory_order_relaxed);
        const uint64_t job = (ticket_.load(std::memory_order_relaxed) >> 32) + 1;
        ticket_.store(job << 32 | static_cast<uint64_t>(n) << 16, std::memory_order_seq_cst);
        if (sleepers_.load(std::memory_order_seq_cst) > 0) {
            std::lock_guard<std::mutex> lock(mu_);
            cv_.notify_all();
        }
        while (take()) {}   // the caller helps
        while (pending_.load(std::memory_order_acquire) != 0) relax();
    }

private:
    static constexpr int kMaxSlices = 0xFFFF;
    HostPool() {
        unsigned hw = std::thread::hardware_concurrency();
        unsigned want = std::min(hw ? hw / 2 : 2u, 8u);
        if (const char *env = std::getenv("SDDMM_B200_HOST_THREADS")) {   // override: 1 .. 64 threads including the caller
            const int v = std::atoi(env);
            if (v >= 1 && v <= 64) want = static_cast<unsigned>(v);
        }
        const int n = static_cast<int>(std::max(1u, want)) - 1;
        for (int i = 0; i < n; ++i) workers_.emplace_back([this] { loop(); });
    }
    ~HostPool() {
        {
            std::lock_guard<std::mutex> lock(mu_);
            stop_.store(true);
        }
        cv_.notify_all();
        for (std::thread &t : workers_) t.join();
    }
    static void relax() {
#if defined(__SSE2__)
        _mm_pause();
#else
        std::this_thread::yield();
#endif
    }
    static bool open(uint64_t t) { return (t & 0xFFFF) < ((t >> 16) & 0xFFFF); }
    // run one slice of the current job, if one is left
    bool take() {
        uint64_t t = ticket_.load(std::memory_order_acquire);
        do {
            if (!open(t)) return false;
        } while (!ticket_.compare_exchange_weak(t, t + 1, std::memory_order_acq_rel, std::memory_order_acquire));
        (*job_)(static_cast<int>(t & 0xFFFF));   // (the job cannot end before this slice has been counted off)
        pending_.fetch_sub(1, std::memory_order_acq_rel);
        return true;
    }
    void loop() {
        while (!stop_.load(std::memory_order_relaxed)) {
            while (take()) {}
            const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(200);
            bool found = false;
            while (!found && std::chrono::steady_clock::now() < until) {
                for (int i = 0; i < 64 && !found; ++i) {
                    relax();
                    found = open(ticket_.load(std::memory_order_acquire));
                }
            }
            if (found) continue;
            std::unique_lock<std::mutex> lock(mu_);
            sleepers_.fetch_add(1, std::memory_order_seq_cst);
            cv_.wait(lock, [&] { return stop_.load() || open(ticket_.load(std::memory_order_seq_cst)); });
            sleepers_.fetch_sub(1, std::memory_order_seq_cst);
        }
    }
    std::vector<std::thread> workers_;
    std::mutex mu_, run_mu_;
    std::condition_variable cv_;
    const std::function<void(int)> *job_ = nullptr;
    std::atomic<uint64_t> ticket_{0};   // job << 32 | slices << 16 | next slice
    std::atomic<int> pending_{0}, sleepers_{0};
    std::atomic<bool> stop_{false};
};

// memcpy whose stores bypass the cache (x86): the destination is a pinned staging buffer that the DMA engine reads next,
// no host thread does, so write-allocating its lines would only add a read of memory per line written.
// SDDMM_B200_STREAM_STORES=0 switches back to plain memcpy.
inline void stream_copy(void *dst, const void *src, size_t bytes) {
#if defined(__SSE2__)
    static const bool enabled = [] { const char *e = std::getenv("SDDMM_B200_STREAM_STORES"); return !(e && e[0] == '0'); }();
    char *d = static_cast<char *>(dst);
    const char *s = static_cast<const char *>(src);
    if (enabled && bytes >= 4096 && (reinterpret_cast<uintptr_t>(d) & 15) == 0) {
        size_t n = bytes / 64;
        for (; n; --n, d += 64, s += 64) {
            const __m128i a = _mm_loadu_si128(reinterpret_cast<const __m128i *>(s));
            const __m128i b = _mm_loadu_si128(reinterpret_cast<const __m128i *>(s + 16));
            const __m128i c = _mm_loadu_si128(reinterpret_cast<const __m128i *>(s + 32));
            const __m128i e = _mm_loadu_si128(reinterpret_cast<const __m128i *>(s + 48));
            _mm_stream_si128(reinterpret_cast<__m128i *>(d), a);
            _mm_stream_si128(reinterpret_cast<__m128i *>(d + 16), b);
            _mm_stream_si128(reinterpret_cast<__m128i *>(d + 32), c);
            _mm_stream_si128(reinterpret_cast<__m128i *>(d + 48), e);
        }
        _mm_sfence();
        bytes &= 63;
    }
    if (bytes) std::memcpy(d, s, bytes);
#else
    std::memcpy(dst, src, bytes);
#endif
}

inline void parallel_memcpy(void *dst, const void *src, size_t bytes, bool stream_stores = false) {
    HostPool &pool = HostPool::instance();
    const int parts = static_cast<int>(std::min<size_t>(pool.width(), std::max<size_t>(1, bytes >> 17)));   // >= 128 KiB per slice
    if (parts <= 1) {
        if (stream_stores) stream_copy(dst, src, bytes); else std::memcpy(dst, src, bytes);
        return;
    }
    const size_t per = (bytes / parts + 4095) & ~size_t(4095);
    pool.run(parts, [&](int k) {
        const size_t off = std::min(bytes, per * static_cast<size_t>(k));
        const size_t len = std::min(per, bytes - off);
        if (!len) return;
        if (stream_stores) stream_copy(static_cast<char *>(dst) + off, static_cast<const char *>(src) + off, len);
        else std::memcpy(static_cast<char *>(dst) + off, static_cast<const char *>(src) + off, len);
    });
}

// Pinned buffers outlive the engine that asked for them (allocating one takes 0.3 ms at best and tens of ms on a busy host):
// at most kMost are kept, and the last engine gives them all back.  A buffer is returned only when its copies have finished.
class PinnedPool {
public:
    static constexpr size_t kMost = 12;   // two rings of two engines
    static PinnedPool &instance() {
        static PinnedPool *pool = new PinnedPool();   // (never destroyed: engines of static storage may end after it would be)
        return *pool;
    }
    void add_user() {
        std::lock_guard<std::mutex> lock(mu_);
        ++users_;
    }
    void remove_user() {
        std::lock_guard<std::mutex> lock(mu_);
        if (--users_ > 0) return;
        for (char *p : free_) cudaFreeHost(p);
        free_.clear();
    }
    char *take(size_t bytes) {
        {
            std::lock_guard<std::mutex> lock(mu_);
            if (bytes == size_ && !free_.empty()) {
                char *p = free_.back();
                free_.pop_back();
                return p;
            }
        }
        void *p = nullptr;
        if (cudaHostAlloc(&p, bytes, cudaHostAllocPortable) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        return static_cast<char *>(p);
    }
    void put(char *p, size_t bytes) {
        {
            std::lock_guard<std::mutex> lock(mu_);
            if (free_.empty()) size_ = bytes;   // (one size at a time: that of the last ring)
            if (users_ > 0 && bytes == size_ && free_.size() < kMost) {
                free_.push_back(p);
                return;
            }
        }
        cudaFreeHost(p);
    }

private:
    std::mutex mu_;
    std::vector<char *> free_;
    size_t size_ = 0;
    int users_ = 0;
};

// a ring of pinned buffers of one engine
struct HostStager {
    // bytes per piece (= size of each pinned buffer); SDDMM_B200_STAGE_MB overrides the 4 MiB default (1 .. 256).
    const size_t kPiece = [] {
        size_t mb = 4;
        if (const char *env = std::getenv("SDDMM_B200_STAGE_MB")) {
            const int v = std::atoi(env);
            if (v >= 1 && v <= 256) mb = static_cast<size_t>(v);
        }
        return mb << 20;
    }();
    static constexpr size_t kMinStaged = size_t(512) << 10;   // smaller copies are left to the driver
    static constexpr int kRing = 3;
    char *buf[kRing] = {};
    cudaEvent_t ev[kRing] = {};
    bool busy[kRing] = {};
    int last = kRing - 1;   // buffer the last piece took

    // buffer b of the ring, allocated when it is first used
    bool ready(int b) {
        if (!buf[b]) buf[b] = PinnedPool::instance().take(kPiece);
        if (!ev[b] && cudaEventCreateWithFlags(&ev[b], cudaEventDisableTiming) != cudaSuccess) {
            cudaGetLastError();
            ev[b] = nullptr;
        }
        return buf[b] && ev[b];
    }
    // the buffer for the next piece: one whose copy has finished if the ring has one (an engine of small copies then pins one
    // buffer, not three: pinning 4 MiB costs 1 to 3 ms), else the next of the ring
    int idle() {
        for (int i = 0; i < kRing; ++i) {
            const int b = (last + i) % kRing;
            if (busy[b] && cudaEventQuery(ev[b]) == cudaSuccess) busy[b] = false;
            if (buf[b] && !busy[b]) return last = b;
        }
        cudaGetLastError();   // (cudaErrorNotReady)
        return last = (last + 1) % kRing;
    }
    void release() {
        for (int i = 0; i < kRing; ++i) {
            if (ev[i]) cudaEventSynchronize(ev[i]);
            if (ev[i]) cudaEventDestroy(ev[i]);
            if (buf[i]) PinnedPool::instance().put(buf[i], kPiece);
            ev[i] = nullptr;
            buf[i] = nullptr;
            busy[i] = false;
        }
    }
    static bool pageable(const void *p) {
        cudaPointerAttributes a;
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return a.type == cudaMemoryTypeUnregistered;
    }

    // host -> device on `stream`; the caller's buffer is free when this returns if it was staged
    cudaError_t upload(void *dst, const void *src, size_t bytes, cudaStream_t stream) {
        if (bytes < kMinStaged || !pageable(src)) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, stream);
        for (size_t off = 0; off < bytes; off += kPiece) {
            const size_t len = std::min(kPiece, bytes - off);
            const int b = idle();
            if (!ready(b)) return cudaMemcpyAsync(static_cast<char *>(dst) + off, static_cast<const char *>(src) + off, bytes - off, cudaMemcpyHostToDevice, stream);
            if (busy[b]) {
                const cudaError_t st = cudaEventSynchronize(ev[b]);
                if (st != cudaSuccess) return st;
            }
            parallel_memcpy(buf[b], static_cast<const char *>(src) + off, len, /*stream_stores=*/true);
            cudaError_t st = cudaMemcpyAsync(static_cast<char *>(dst) + off, buf[b], len, cudaMemcpyHostToDevice, stream);
            if (st == cudaSuccess) st = cudaEventRecord(ev[b], stream);
            if (st != cudaSuccess) return st;
            busy[b] = true;
        }
        return cudaSuccess;
    }
    // device -> host on `stream`; returns when the caller's buffer is filled (the stream has drained up to the copy)
    cudaError_t download(void *dst, const void *src, size_t bytes, cudaStream_t stream) {
        const size_t pieces = (bytes + kPiece - 1) / kPiece;
        bool staged = bytes >= kMinStaged && pageable(dst);
        for (int b = 0; staged && b < kRing && static_cast<size_t>(b) < pieces; ++b) staged = ready(b);
        if (!staged) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream);
        for (int b = 0; b < kRing; ++b)
            if (busy[b]) {
                const cudaError_t st = cudaEventSynchronize(ev[b]);
                if (st != cudaSuccess) return st;
                busy[b] = false;
            }
        auto enqueue = [&](size_t c) -> cudaError_t {
            const size_t off = c * kPiece, len = std::min(kPiece, bytes - off);
            cudaError_t st = cudaMemcpyAsync(buf[c % kRing], static_cast<const char *>(src) + off, len, cudaMemcpyDeviceToHost, stream);
            if (st == cudaSuccess) st = cudaEventRecord(ev[c % kRing], stream);
            return st;
        };
        cudaError_t st = cudaSuccess;
        for (size_t c = 0; c < kRing - 1 && c < pieces && st == cudaSuccess; ++c) st = enqueue(c);
        for (size_t c = 0; c < pieces && st == cudaSuccess; ++c) {
            st = cudaEventSynchronize(ev[c % kRing]);                           // piece c has landed in its pinned buffer
            if (st != cudaSuccess) break;
            if (c + kRing - 1 < pieces) st = enqueue(c + kRing - 1);            // later pieces cross the link while this one is copied out
            const size_t off = c * kPiece, len = std::min(kPiece, bytes - off);
            parallel_memcpy(static_cast<char *>(dst) + off, buf[c % kRing], len);
        }
        return st;
    }
};

}  // namespace sddmm
