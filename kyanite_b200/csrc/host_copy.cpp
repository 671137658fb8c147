// One core copies 18 GB/s into pinned memory, a third of what the link to the GPU takes: a 1.4 MB batch of boards was
// 75 us on the caller's thread before its 35 us upload could start.  Four threads and an upload per finished range
// bring the two to about 45 us together.
#include "host_copy.h"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

#ifdef __SSE2__
#include <emmintrin.h>
#endif

namespace kn {

namespace {

// memcpy whose stores bypass the caches.  The helpers' part of a staging buffer would otherwise sit modified in the
// caches of cores that go to sleep right after, and the GPU's read of it took four times as long (1.4 MB: 140 us
// against 35).
void copy_past_caches(uint8_t* dst, const uint8_t* src, size_t bytes) {
#ifdef __SSE2__
    size_t i = 0;
    if (((uintptr_t)dst & 15) == 0) {
        for (; i + 64 <= bytes; i += 64) {
            const __m128i a = _mm_loadu_si128((const __m128i*)(src + i)), b = _mm_loadu_si128((const __m128i*)(src + i + 16));
            const __m128i c = _mm_loadu_si128((const __m128i*)(src + i + 32)), d = _mm_loadu_si128((const __m128i*)(src + i + 48));
            _mm_stream_si128((__m128i*)(dst + i), a);
            _mm_stream_si128((__m128i*)(dst + i + 16), b);
            _mm_stream_si128((__m128i*)(dst + i + 32), c);
            _mm_stream_si128((__m128i*)(dst + i + 48), d);
        }
        _mm_sfence();
    }
    memcpy(dst + i, src + i, bytes - i);
#else
    memcpy(dst, src, bytes);
#endif
}

constexpr int kHelpers = 3;
constexpr size_t kChunk = 128 << 10;   // 7 us of one core: small enough to share out 1 MB, large against a wake

constexpr size_t kReadyBytes = 512 << 10;   // least range handed on before the end: an upload costs some 4 us on its own

class Pool : public CopyPool {
   public:
    ~Pool() override {
        {
            std::lock_guard<std::mutex> lock(mu_);
            stop_ = true;
        }
        wake_.notify_all();
        for (auto& t : threads_) t.join();
    }

    void copy(void* dst, const void* src, size_t bytes, bool past_caches, const std::function<void(size_t, size_t)>& ready) override {
        const size_t chunks = (bytes + kChunk - 1) / kChunk;
        std::unique_lock<std::mutex> mine(user_, std::try_to_lock);
        if (!mine.owns_lock() || bytes < kParallelCopyBytes) {
            for (size_t c = 0; c < chunks; c++) {
                const size_t from = c * kChunk, to = std::min(bytes, from + kChunk);
                memcpy((uint8_t*)dst + from, (const uint8_t*)src + from, to - from);
                if (ready) ready(from, to);
            }
            return;
        }
        auto job = std::make_shared<Job>(dst, src, bytes, chunks, past_caches);
        {
            std::lock_guard<std::mutex> lock(mu_);
            if (threads_.empty()) {
                try {
                    for (int i = 0; i < kHelpers; i++) threads_.emplace_back([this] { help(); });
                } catch (const std::system_error&) {   // no more threads to be had: fewer helpers, or none
                }
            }
            job_ = job;
            generation_++;
        }
        wake_.notify_all();
        size_t done = 0;
        auto advance = [&] {
            size_t upto = done;
            while (upto < chunks && job->complete[upto].load(std::memory_order_acquire)) upto++;
            if (upto == done || (upto < chunks && (upto - done) * kChunk < kReadyBytes)) return;
            if (ready) ready(done * kChunk, std::min(bytes, upto * kChunk));
            done = upto;
        };
        try {
            while (job->one()) advance();
            while (done < chunks) {   // what the helpers still have in hand: a few microseconds
                advance();
                if (done < chunks) std::this_thread::yield();
            }
        } catch (...) {   // from `ready`; the caller is free to drop both buffers once it leaves here
            job->abandon();
            throw;
        }
    }

   private:
    struct Job {
        uint8_t* dst;
        const uint8_t* src;
        size_t bytes, chunks;
        bool past_caches;
        std::atomic<size_t> next{0};
        std::vector<std::atomic<uint8_t>> complete;
        Job(void* d, const void* s, size_t b, size_t c, bool past)
            : dst((uint8_t*)d), src((const uint8_t*)s), bytes(b), chunks(c), past_caches(past), complete(c) {}
        bool one() {
            const size_t c = next.fetch_add(1, std::memory_order_relaxed);
            if (c >= chunks) return false;
            const size_t from = c * kChunk;
            const size_t n = std::min(bytes, from + kChunk) - from;
            if (past_caches) copy_past_caches(dst + from, src + from, n);
            else memcpy(dst + from, src + from, n);
            complete[c].store(1, std::memory_order_release);
            return true;
        }
        // no further chunks are handed out, and those that were are complete
        void abandon() {
            const size_t taken = std::min(next.exchange(chunks), chunks);
            for (size_t c = 0; c < taken; c++)
                while (!complete[c].load(std::memory_order_acquire)) std::this_thread::yield();
        }
    };

    void help() {
        uint64_t seen = 0;
        for (;;) {
            std::shared_ptr<Job> job;
            {
                std::unique_lock<std::mutex> lock(mu_);
                wake_.wait(lock, [&] { return stop_ || generation_ != seen; });
                if (stop_) return;
                seen = generation_;
                job = job_;
            }
            // (a job that is over hands out no more chunks: its buffers are not touched by a helper that wakes late)
            while (job->one()) {
            }
        }
    }

    std::mutex user_;   // held by the caller whose job the helpers work on
    std::mutex mu_;
    std::condition_variable wake_;
    std::vector<std::thread> threads_;
    std::shared_ptr<Job> job_;
    uint64_t generation_ = 0;
    bool stop_ = false;
};

}  // namespace

std::shared_ptr<CopyPool> CopyPool::shared() {
    static std::mutex mu;
    static std::weak_ptr<CopyPool> existing;
    std::lock_guard<std::mutex> lock(mu);
    std::shared_ptr<CopyPool> p = existing.lock();
    if (!p) existing = p = std::make_shared<Pool>();
    return p;
}

}  // namespace kn
