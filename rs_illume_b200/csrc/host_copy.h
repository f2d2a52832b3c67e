// Staging of pageable host memory: a pinned block, and copies on several threads.
//
// A query on pageable buffers is bound by the host's copies: one thread moves
// about 10 GB/s, and the driver's own staging of pageable memory is one
// thread's.  Blocks of a copy are handed out by a counter to the calling
// thread and up to seven helpers, which sleep between calls and spin for a
// moment between the copies of one call.
#pragma once
#include <cuda_runtime.h>
#include <unistd.h>

#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <memory>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace ilm {

class HostCopier {
public:
    HostCopier() {
        const unsigned hw = std::thread::hardware_concurrency();
        const unsigned helpers = hw / 2 < 7 ? hw / 2 : 7;
        try {
            for (unsigned k = 0; k < helpers; ++k) threads_.emplace_back([this] { helper(); });
        } catch (const std::system_error&) {
            // fewer helpers, or none: the caller copies alone
        }
    }
    ~HostCopier() {
        if (getpid() != owner_) {   // a forked child has no helpers to stop or join
            for (auto& t : threads_) t.detach();
            return;
        }
        {
            std::lock_guard<std::mutex> lock(mu_);
            stop_.store(true, std::memory_order_relaxed);
        }
        wake_.notify_all();
        for (auto& t : threads_) t.join();
    }
    HostCopier(const HostCopier&) = delete;
    HostCopier& operator=(const HostCopier&) = delete;

    // Returns when all `bytes` are copied.  One caller at a time.
    void copy(void* dst, const void* src, size_t bytes) {
        auto job = std::make_shared<Job>();
        job->dst = static_cast<char*>(dst);
        job->src = static_cast<const char*>(src);
        job->bytes = bytes;
        job->blocks = (bytes + kBlock - 1) / kBlock;
        if (!threads_.empty() && job->blocks > 1) {
            {
                std::lock_guard<std::mutex> lock(mu_);
                job_ = job;
                generation_.fetch_add(1, std::memory_order_relaxed);
            }
            wake_.notify_all();
        }
        job->work();
        while (job->done.load(std::memory_order_acquire) != job->blocks) std::this_thread::yield();
    }

private:
    static constexpr size_t kBlock = 64 << 10;
    static constexpr int kSpins = 4000;   // a few tens of microseconds

    // A helper that comes late works on a job of its own reference, which has
    // no blocks left.
    struct Job {
        char* dst = nullptr;
        const char* src = nullptr;
        size_t bytes = 0, blocks = 0;
        std::atomic<size_t> next{0}, done{0};
        void work() {
            for (size_t b; (b = next.fetch_add(1, std::memory_order_relaxed)) < blocks;) {
                const size_t at = b * kBlock;
                std::memcpy(dst + at, src + at, bytes - at < kBlock ? bytes - at : kBlock);
                done.fetch_add(1, std::memory_order_release);
            }
        }
    };

    void helper() {
        uint64_t seen = 0;
        for (;;) {
            for (int k = 0; k < kSpins && generation_.load(std::memory_order_relaxed) == seen &&
                            !stop_.load(std::memory_order_relaxed);
                 ++k)
                pause();
            std::shared_ptr<Job> job;
            {
                std::unique_lock<std::mutex> lock(mu_);
                wake_.wait(lock, [&] {
                    return stop_.load(std::memory_order_relaxed) ||
                           generation_.load(std::memory_order_relaxed) != seen;
                });
                if (stop_.load(std::memory_order_relaxed)) return;
                seen = generation_.load(std::memory_order_relaxed);
                job = job_;
            }
            job->work();
        }
    }
    static void pause() {
#if defined(__x86_64__)
        __builtin_ia32_pause();
#endif
    }

    const pid_t owner_ = getpid();
    std::vector<std::thread> threads_;
    std::mutex mu_;
    std::condition_variable wake_;
    std::shared_ptr<Job> job_;
    std::atomic<uint64_t> generation_{0};
    std::atomic<bool> stop_{false};
};

// One context's staging.  `block` is null if the memory could not be pinned.
struct HostStaging {
    static constexpr size_t kBlockBytes = 8ull << 20;
    void* block = nullptr;
    HostCopier copier;

    HostStaging() {
        if (cudaHostAlloc(&block, kBlockBytes, cudaHostAllocDefault) != cudaSuccess) {
            cudaGetLastError();
            block = nullptr;
        }
    }
    ~HostStaging() {
        if (block) cudaFreeHost(block);
    }
    HostStaging(const HostStaging&) = delete;
    HostStaging& operator=(const HostStaging&) = delete;
};

}  // namespace ilm
