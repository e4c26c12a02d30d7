// fy_hostcopy.h -- copies between a caller's pageable memory and the device through pinned staging,
// the host side spread over a few threads.
//
// A pageable cudaMemcpyAsync runs at the speed of one core's memcpy (8.4 MB in 0.49 ms here, 17 GB/s)
// while the link takes 0.16 ms. Here a copy is cut into chunks: helper threads move chunks between the
// caller's memory and a pinned ring, the calling thread queues each chunk's DMA as it becomes ready
// (to the device) or hands it on as it lands (from the device), and moves chunks itself in between.
// One fy_deconvolve after another, plain / staged: 8x512x512 floats 940 / 765 us, 16x512x512 1800 / 1170,
// 256^3 9.5 / 4.4 ms; 1 and 2 MB are faster plain (190 / 250 us, 300 / 335), so staging begins at 4.
// Helpers live for one call and are joined in it. They look for work without sleeping, since waking a
// sleeping core costs more than a chunk (with helpers that sleep whenever there is none, the slab took
// 1300 us), but only for kSpin at a time: while the GPU works longer, they sleep.
// All callers together have at most half the cores as helpers, and beyond a quarter of the cores in
// callers the next one copies plainly, since plain copies of as many callers fill the link by
// themselves. Plain / staged / staged without that limit on 16 cores, us a call of 8 MB: 2 callers
// 556 / 422 / 417, 4: 786 / 642 / 762, 8: 986 / 833 / 962, 16: 1049 / 942 / 1115. The time is bought with
// helpers' CPU time: 0.95 ms a call plain, 4.2 ms staged with one caller, 1.8 and 2.0 ms with 16.
// Without helpers, without pinned memory and for a caller's buffer that is not pageable host memory
// (pinned, managed, on a device) the plain copies run.
#pragma once
#include <string.h>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <mutex>
#include <thread>
#include <vector>
#include "fy_context.h"

namespace fy {

class HostCopy {
public:
    static constexpr size_t kChunk = 1 << 20, kRing = 16 << 20, kMin = 4 << 20;
    static constexpr int kSlots = (int)(kRing / kChunk), kHelpers = 5;
    static constexpr std::chrono::microseconds kSpin{1000};

    // For a call that copies `bytes` from `in` to the device and back to `out`: which of the two are
    // staged, and what that takes (nothing where neither is).
    HostCopy(size_t bytes, const void* in, const void* out) {
        if (bytes < kMin) return;
        const bool up = is_pageable(in), down = is_pageable(out);
        if (!up && !down) return;
        counted_ = true;
        const int hw = (int)std::thread::hardware_concurrency();
        if (callers().fetch_add(1) >= hw / 4) return;
        while (mine_ < kHelpers && helpers().fetch_add(1) < hw / 2) ++mine_;
        if (mine_ < kHelpers) helpers().fetch_sub(1);
        if (mine_ == 0 || ctx().pin2.ensure(kRing) != cudaSuccess) return;
        const int n = !down ? 0 : bytes < kRing ? chunks_of(bytes) : kSlots;
        for (int i = 0; i < n; ++i)
            if (cudaEventCreateWithFlags(&ev_[i], cudaEventDisableTiming) != cudaSuccess) {
                cudaGetLastError();
                return;
            }
        up_ = up;
        down_ = down;
    }
    ~HostCopy() {
        {
            std::lock_guard<std::mutex> lk(mu_);
            quit_.store(true, std::memory_order_release);
        }
        cv_.notify_all();
        for (auto& t : th_) t.join();
        helpers().fetch_sub(mine_);
        if (counted_) callers().fetch_sub(1);
        for (auto& e : ev_)
            if (e) cudaEventDestroy(e);
    }
    HostCopy(const HostCopy&) = delete;

    cudaError_t to_device(void* dst, const void* src, size_t bytes, cudaStream_t st) {
        if (!up_) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
        char* ring = (char*)ctx().pin2.p;
        for (size_t at = 0; at < bytes; at += kRing) {
            const size_t n = bytes - at < kRing ? bytes - at : kRing;
            cudaError_t e = cudaSuccess;
            if (at && (e = cudaStreamSynchronize(st)) != cudaSuccess) return e;      // the ring is read out
            const int chunks = begin(ring, (const char*)src + at, n, chunks_of(n));
            for (int i = 0; i < chunks && e == cudaSuccess; ++i) {
                while (!done_[i].load(std::memory_order_acquire))
                    if (!move_one()) std::this_thread::yield();
                const size_t o = (size_t)i * kChunk, m = n - o < kChunk ? n - o : kChunk;
                e = cudaMemcpyAsync((char*)dst + at + o, ring + o, m, cudaMemcpyHostToDevice, st);
            }
            finish(chunks);
            if (e != cudaSuccess) return e;
        }
        return cudaSuccess;
    }
    // Returns with the data in dst (the stream is waited for).
    cudaError_t from_device(void* dst, const void* src, size_t bytes, cudaStream_t st) {
        if (!down_) {
            const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
            return e != cudaSuccess ? e : cudaStreamSynchronize(st);
        }
        char* ring = (char*)ctx().pin2.p;
        for (size_t at = 0; at < bytes; at += kRing) {
            const size_t n = bytes - at < kRing ? bytes - at : kRing;
            const int chunks = chunks_of(n);
            cudaError_t e = cudaSuccess;
            for (int i = 0; i < chunks && e == cudaSuccess; ++i) {
                const size_t o = (size_t)i * kChunk, m = n - o < kChunk ? n - o : kChunk;
                e = cudaMemcpyAsync(ring + o, (const char*)src + at + o, m, cudaMemcpyDeviceToHost, st);
                if (e == cudaSuccess) e = cudaEventRecord(ev_[i], st);
            }
            if (e != cudaSuccess) {
                cudaStreamSynchronize(st);               // nothing of this call is left in flight
                return e;
            }
            begin((char*)dst + at, ring, n, 0);
            for (int i = 0; i < chunks && e == cudaSuccess; ++i) {
                e = cudaEventSynchronize(ev_[i]);
                if (e == cudaSuccess) show(i + 1);
            }
            if (e != cudaSuccess) {
                stop();
                return e;
            }
            while (move_one()) {}
            finish(chunks);
        }
        return cudaSuccess;
    }

private:
    static int chunks_of(size_t n) { return (int)((n + kChunk - 1) / kChunk); }
    static std::atomic<int>& callers() {
        static std::atomic<int> n{0};
        return n;
    }
    static std::atomic<int>& helpers() {
        static std::atomic<int> n{0};
        return n;
    }
    // A job: chunks [0, ready_) of n bytes may be moved from `from` to `to`. Helpers enter it through
    // open_ and are counted in inside_ while they may look at it. One that finds nothing to move for
    // kSpin sleeps until there is.
    int begin(char* to, const char* from, size_t n, int ready) {
        to_ = to;
        from_ = from;
        n_ = n;
        chunks_ = chunks_of(n);
        for (int i = 0; i < chunks_; ++i) done_[i].store(false, std::memory_order_relaxed);
        next_.store(0, std::memory_order_relaxed);
        ready_.store(0, std::memory_order_relaxed);
        open_.store(true, std::memory_order_seq_cst);
        show(ready);
        while ((int)th_.size() < mine_) {                // the first job starts while they start
            try {
                th_.emplace_back([this] { help(); });
            } catch (...) {                              // no thread to be had: fewer helpers, or this one alone
                helpers().fetch_sub(mine_ - (int)th_.size());
                mine_ = (int)th_.size();
            }
        }
        return chunks_;
    }
    // Closes the job once its chunks are moved (all of them have been claimed by then).
    void finish(int chunks) {
        for (int i = 0; i < chunks; ++i)
            while (!done_[i].load(std::memory_order_acquire))
                if (!move_one()) std::this_thread::yield();
        stop();
    }
    void stop() {
        open_.store(false, std::memory_order_seq_cst);
        while (inside_.load(std::memory_order_seq_cst)) std::this_thread::yield();
    }
    // Raises ready_. Under mu_, so that a helper about to sleep sees it or is woken.
    void show(int ready) {
        {
            std::lock_guard<std::mutex> lk(mu_);
            ready_.store(ready, std::memory_order_release);
        }
        cv_.notify_all();
    }
    bool move_one() {
        int i = next_.load(std::memory_order_relaxed);
        do {
            if (i >= ready_.load(std::memory_order_acquire)) return false;
        } while (!next_.compare_exchange_weak(i, i + 1, std::memory_order_acq_rel));
        const size_t o = (size_t)i * kChunk, m = n_ - o < kChunk ? n_ - o : kChunk;
        memcpy(to_ + o, from_ + o, m);
        done_[i].store(true, std::memory_order_release);
        return true;
    }
    // looks without writing until there is something to move
    bool work() const {
        return open_.load(std::memory_order_acquire) &&
               next_.load(std::memory_order_relaxed) < ready_.load(std::memory_order_relaxed);
    }
    void help() {
        while (!quit_.load(std::memory_order_acquire)) {
            const auto until = std::chrono::steady_clock::now() + kSpin;
            bool found = false;
            while (!(found = work()) && !quit_.load(std::memory_order_acquire) && std::chrono::steady_clock::now() < until)
                std::this_thread::yield();
            if (found) {
                inside_.fetch_add(1, std::memory_order_seq_cst);
                if (open_.load(std::memory_order_seq_cst)) move_one();
                inside_.fetch_sub(1, std::memory_order_seq_cst);
            } else {
                std::unique_lock<std::mutex> lk(mu_);
                cv_.wait(lk, [this] { return quit_.load(std::memory_order_relaxed) || work(); });
            }
        }
    }

    char* to_ = nullptr;
    const char* from_ = nullptr;
    size_t n_ = 0;
    int chunks_ = 0;
    std::atomic<int> next_{0}, ready_{0}, inside_{0};
    std::atomic<bool> open_{false}, quit_{false};
    std::atomic<bool> done_[kSlots];
    std::mutex mu_;
    std::condition_variable cv_;
    cudaEvent_t ev_[kSlots] = {};
    std::vector<std::thread> th_;
    int mine_ = 0;                                       // helpers of the common allowance that are this call's
    bool counted_ = false;                               // among the callers
    bool up_ = false, down_ = false;                     // staged to, from the device
};

}  // namespace fy
