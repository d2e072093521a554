// Uploads of camera frames from ordinary (pageable) host memory.
//
// The driver copies pageable memory through a staging buffer of its own on the calling thread: 294 us for a 5 MB frame and
// 1.14 ms for a 21 MB one on a B200's host of 16 cores, against 102 us and 400 us of bus time. Here the frame is cut into slices
// that the calling thread and a few helper threads copy into the lane's pinned buffer with non-temporal stores (which leave no
// dirty lines for the bus to snoop), and every run of finished slices is sent on its way while the next ones are copied: 143 us
// and 504 us. The helpers sleep between uploads; they belong to all engines of the process, and the last engine ends them.
#pragma once

#include <cuda_runtime.h>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <exception>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

#include "conv_dispatch.hpp"

namespace vm {

// bytes per slice: 64 KB slices measured 15-35 % slower (more copies to issue), 1 MB slices 10-35 % (the first one starts late)
constexpr size_t UPLOAD_SLICE = 256 << 10;
// a run of finished slices is sent when it has this many bytes (an asynchronous copy costs 2-3 us to issue)
constexpr size_t UPLOAD_RUN = 512 << 10;
// with two helpers 5 MB take 143 us, with one 157 and with none 281; a third gains 3 us
constexpr int UPLOAD_HELPERS = 2;

inline void copy_past_the_cache(uint8_t* dst, const uint8_t* src, size_t n) {
#if defined(__SSE2__)
    const size_t head = std::min(n, (16 - (reinterpret_cast<uintptr_t>(dst) & 15)) & 15);
    std::memcpy(dst, src, head);
    size_t i = head;
    for (; i + 64 <= n; i += 64) {
        const __m128i a = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i));
        const __m128i b = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i + 16));
        const __m128i c = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i + 32));
        const __m128i d = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i + 48));
        _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i), a);
        _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i + 16), b);
        _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i + 32), c);
        _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i + 48), d);
    }
    std::memcpy(dst + i, src + i, n - i);
    _mm_sfence();
#else
    std::memcpy(dst, src, n);  // other hosts
#endif
}

struct UploadSlice {
    const uint8_t* src;
    size_t offset;  // in the staging buffer and in the device buffer
    size_t bytes;
};

// The slices of one chunk's frames, claimed one by one by whoever is free.
struct UploadJob {
    std::vector<UploadSlice> slices;
    std::vector<std::atomic<uint8_t>> done;
    std::atomic<size_t> next{0};
    std::atomic<int> helpers{0};  // helpers at work on this job
    uint8_t* staging = nullptr;

    void add(const uint8_t* src, size_t offset, size_t bytes) {
        for (size_t at = 0; at < bytes; at += UPLOAD_SLICE) slices.push_back({src + at, offset + at, std::min(UPLOAD_SLICE, bytes - at)});
    }
    void arm(uint8_t* to) {
        staging = to;
        done    = std::vector<std::atomic<uint8_t>>(slices.size());
        next    = 0;
    }
    bool copy_one() {
        const size_t i = next.fetch_add(1);
        if (i >= slices.size()) return false;
        copy_past_the_cache(staging + slices[i].offset, slices[i].src, slices[i].bytes);
        done[i].store(1, std::memory_order_release);
        return true;
    }
};

class UploadHelpers {
public:
    static std::shared_ptr<UploadHelpers> get() {
        static std::mutex mutex;
        static std::weak_ptr<UploadHelpers> shared;
        std::lock_guard<std::mutex> lock(mutex);
        std::shared_ptr<UploadHelpers> h = shared.lock();
        if (!h) {
            h.reset(new UploadHelpers());
            shared = h;
        }
        return h;
    }
    ~UploadHelpers() {
        {
            std::lock_guard<std::mutex> lock(mutex_);
            stop_ = true;
        }
        wake_.notify_all();
        for (auto& t : threads_) t.join();
    }
    // Offers a job to the helpers; one at a time, an engine that finds them busy copies alone.
    bool offer(UploadJob* job) {
        {
            std::lock_guard<std::mutex> lock(mutex_);
            if (job_ != nullptr || threads_.empty()) return false;
            job_ = job;
            ++generation_;
        }
        wake_.notify_all();
        return true;
    }
    // Takes an offered job back; returns when no helper touches it any more (at most the copy of one slice later).
    void withdraw(UploadJob* job) {
        {
            std::lock_guard<std::mutex> lock(mutex_);
            if (job_ == job) job_ = nullptr;
        }
        while (job->helpers.load(std::memory_order_acquire) != 0) std::this_thread::yield();
    }

private:
    UploadHelpers() {
        const int n = std::min<int>(UPLOAD_HELPERS, static_cast<int>(std::thread::hardware_concurrency()) / 4);
        threads_.reserve(UPLOAD_HELPERS);
        try {
            for (int i = 0; i < n; ++i) threads_.emplace_back([this] { work(); });
        }
        catch (const std::exception&) {}  // a limit on threads: those that did start help, and an upload without any copies alone
    }
    void work() {
        uint64_t seen = 0;
        for (;;) {
            UploadJob* job = nullptr;
            {
                std::unique_lock<std::mutex> lock(mutex_);
                wake_.wait(lock, [&] { return stop_ || generation_ != seen; });
                if (stop_) return;
                seen = generation_;
                job  = job_;
                if (job == nullptr) continue;
                job->helpers.fetch_add(1);
            }
            while (job->copy_one()) {}
            job->helpers.fetch_sub(1, std::memory_order_release);
        }
    }
    std::mutex mutex_;
    std::condition_variable wake_;
    std::vector<std::thread> threads_;
    UploadJob* job_      = nullptr;
    uint64_t generation_ = 0;
    bool stop_           = false;
};

// One chunk's upload under way: the calling thread pumps it between its other work and finishes it before the chunk's images are
// sampled.
class Upload {
public:
    Upload(UploadHelpers* helpers, uint8_t* device, cudaStream_t stream) : helpers_(helpers), device_(device), stream_(stream) {}
    ~Upload() {
        if (offered_) helpers_->withdraw(&job);
    }
    Upload(const Upload&) = delete;
    Upload& operator=(const Upload&) = delete;

    UploadJob job;

    void start(uint8_t* staging) {
        job.arm(staging);
        if (job.slices.size() > 1 && helpers_ != nullptr) offered_ = helpers_->offer(&job);
    }
    // sends what is ready
    void pump(bool all = false) {
        size_t to = issued_;
        while (to < job.slices.size() && job.done[to].load(std::memory_order_acquire)) ++to;
        if (to == issued_) return;
        const size_t begin = job.slices[issued_].offset;
        const size_t end   = job.slices[to - 1].offset + job.slices[to - 1].bytes;
        if (end - begin < UPLOAD_RUN && to < job.slices.size() && !all) return;
        VM_CUDA(cudaMemcpyAsync(device_ + begin, job.staging + begin, end - begin, cudaMemcpyHostToDevice, stream_));
        issued_ = to;
    }
    void finish() {
        while (job.copy_one()) pump();
        while (issued_ < job.slices.size()) pump(true);
        if (offered_) helpers_->withdraw(&job);
        offered_ = false;
    }

private:
    UploadHelpers* helpers_;
    uint8_t* device_;
    cudaStream_t stream_;
    size_t issued_ = 0;
    bool offered_  = false;
};

}  // namespace vm
