// Staging of pageable host memory: a pinned block, and copies on several threads.
//
// A query on pageable buffers is bound by the host's copies: one thread moves
// about 10 GB/s, and the driver's own staging of pageable memory is one
// thread's.  Blocks of a copy are handed out by a counter to the calling
// thread and up to seven helpers, which sleep between calls and spin for a
// moment between the copies of one call.
#pragma once
#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>

#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <exception>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

namespace ilm {

class HostCopier {
public:
    HostCopier() : s_(new State) {
        const unsigned hw = std::thread::hardware_concurrency();
        const unsigned helpers = hw / 2 < 7 ? hw / 2 : 7;
        try {
            s_->threads.reserve(helpers);   // so that a started thread always has its place
            for (unsigned k = 0; k < helpers; ++k) s_->threads.emplace_back([s = s_] { s->helper(); });
        } catch (const std::exception&) {
            // no thread or no memory: fewer helpers, or none: the caller copies alone
        }
    }
    ~HostCopier() {
        // A forked child has no helpers to stop or join, and neither the lock
        // nor the condition variable that they slept on can be destroyed
        // there (it would wait for its sleepers): the state stays.
        if (getpid() != owner_) return;
        {
            std::lock_guard<std::mutex> lock(s_->mu);
            s_->stop.store(true, std::memory_order_relaxed);
        }
        s_->wake.notify_all();
        for (auto& t : s_->threads) t.join();
        delete s_;
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
        if (!s_->threads.empty() && job->blocks > 1) {
            {
                std::lock_guard<std::mutex> lock(s_->mu);
                s_->job = job;
                s_->generation.fetch_add(1, std::memory_order_relaxed);
            }
            s_->wake.notify_all();
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

    struct State {
        std::vector<std::thread> threads;
        std::mutex mu;
        std::condition_variable wake;
        std::shared_ptr<Job> job;
        std::atomic<uint64_t> generation{0};
        std::atomic<bool> stop{false};

        void helper() {
            uint64_t seen = 0;
            for (;;) {
                for (int k = 0; k < kSpins && generation.load(std::memory_order_relaxed) == seen &&
                                !stop.load(std::memory_order_relaxed);
                     ++k)
                    pause();
                std::shared_ptr<Job> mine;
                {
                    std::unique_lock<std::mutex> lock(mu);
                    wake.wait(lock, [&] {
                        return stop.load(std::memory_order_relaxed) ||
                               generation.load(std::memory_order_relaxed) != seen;
                    });
                    if (stop.load(std::memory_order_relaxed)) return;
                    seen = generation.load(std::memory_order_relaxed);
                    mine = job;
                }
                mine->work();
            }
        }
    };
    static void pause() {
#if defined(__x86_64__)
        __builtin_ia32_pause();
#endif
    }

    State* const s_;
    const pid_t owner_ = getpid();
};

// One context's staging: a pinned block on large pages where the system gives
// them, and the copying threads.  If the memory cannot be had, `block` and
// `copier` are null.
//
// Making it is part of some query, so it has to be quick: 8 MB as four large
// pages are touched in 0.8 ms and registered in 0.5; cudaHostAlloc of the same
// takes 4.5 to 4.9 ms, registering 2,048 small pages 4 to 8.
struct HostStaging {
    static constexpr size_t kBlockBytes = 8ull << 20;
    std::unique_ptr<HostCopier> copier;
    void* block = nullptr;

    HostStaging() {
        void* const p = mmap(nullptr, kBlockBytes + kLargePage, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
        if (p == MAP_FAILED) return;
        mapped_ = p;
        void* const at = reinterpret_cast<void*>((reinterpret_cast<uintptr_t>(p) + kLargePage - 1) / kLargePage * kLargePage);
        madvise(at, kBlockBytes, MADV_HUGEPAGE);
        madvise(mapped_, kBlockBytes + kLargePage, MADV_DONTFORK);
        if (cudaHostRegister(at, kBlockBytes, cudaHostRegisterDefault) != cudaSuccess) {
            cudaGetLastError();
            return;
        }
        try {
            copier.reset(new HostCopier());
        } catch (...) {
            cudaHostUnregister(at);
            munmap(mapped_, kBlockBytes + kLargePage);
            throw;
        }
        block = at;
    }
    ~HostStaging() {
        if (getpid() != owner_) return;   // not mapped in a forked child
        if (block) cudaHostUnregister(block);
        if (mapped_) munmap(mapped_, kBlockBytes + kLargePage);
    }
    HostStaging(const HostStaging&) = delete;
    HostStaging& operator=(const HostStaging&) = delete;

private:
    static constexpr size_t kLargePage = 2ull << 20;
    void* mapped_ = nullptr;
    const pid_t owner_ = getpid();
};

}  // namespace ilm
