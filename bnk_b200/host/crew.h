// Threads of the dispatcher: one worker per GPU, and helpers that share the copies of a GPU's share of a call.
#pragma once

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <exception>
#include <functional>
#include <mutex>
#include <queue>
#include <thread>
#include <vector>

#include "../../include/bnk_gpu.h"

namespace crew {

// One host thread per GPU: runs the jobs posted to it in order.  Throws if there is no thread to be had.
class Worker {
  public:
    Worker() : thread_([this] { Run(); }) {}
    ~Worker() {
        {
            std::lock_guard<std::mutex> g(mu_);
            stop_ = true;
        }
        cv_.notify_all();
        thread_.join();
    }
    void Post(std::function<void()> job) {
        {
            std::lock_guard<std::mutex> g(mu_);
            jobs_.push(std::move(job));
        }
        cv_.notify_all();
    }

  private:
    void Run() {
        for (;;) {
            std::function<void()> job;
            {
                std::unique_lock<std::mutex> g(mu_);
                cv_.wait(g, [this] { return stop_ || !jobs_.empty(); });
                if (jobs_.empty()) return;
                job = std::move(jobs_.front());
                jobs_.pop();
            }
            job();
        }
    }
    std::mutex mu_;
    std::condition_variable cv_;
    std::queue<std::function<void()>> jobs_;
    bool stop_ = false;
    std::thread thread_;
};

// counts the per-GPU jobs of one call down
class Latch {
  public:
    explicit Latch(int n) : left_(n) {}
    void Done() {
        std::lock_guard<std::mutex> g(mu_);
        if (--left_ == 0) cv_.notify_all();
    }
    void Wait() {
        std::unique_lock<std::mutex> g(mu_);
        cv_.wait(g, [this] { return left_ <= 0; });
    }

  private:
    std::mutex mu_;
    std::condition_variable cv_;
    int left_;
};

inline void Pause() {
#if defined(__x86_64__) || defined(__i386__)
    __builtin_ia32_pause();
#else
    std::this_thread::yield();
#endif
}

// Work of one thread that others may join.
struct Task {
    virtual ~Task() = default;
    virtual int Drive() = 0; // the calling thread; returns when all is done
    virtual void Help() = 0; // any other
};

// f(first, last) over [0, n) in stretches, whoever is free taking the next one.
struct Stretches : Task {
    static constexpr uint32_t kStretch = 512;
    const uint32_t n;
    const std::function<void(uint32_t, uint32_t)> f;
    std::atomic<uint32_t> next{0}, done{0};
    Stretches(uint32_t n_, std::function<void(uint32_t, uint32_t)> f_) : n(n_), f(std::move(f_)) {}
    int Drive() override {
        Help();
        for (uint32_t idle = 0; done.load(std::memory_order_acquire) < n;) {
            if (++idle < 4000) Pause();
            else std::this_thread::yield();
        }
        return BNK_SUCCESS;
    }
    void Help() override {
        for (;;) {
            const uint32_t at = next.fetch_add(kStretch, std::memory_order_relaxed);
            if (at >= n) return;
            const uint32_t to = std::min(n, at + kStretch);
            f(at, to);
            done.fetch_add(to - at, std::memory_order_release);
        }
    }
};

// A GPU's share of one call in pieces: while one piece is on the GPU the next is copied into the pinned ring of another
// batch and the one before is copied out, by several threads.  (One batch, one thread, one step after the other: 24,576 x
// 1420 B sealed and opened in 21.8 ms, of which the GPU worked 3.)
struct Share : Task {
    static constexpr uint32_t kSlots = 4;  // pinned batches in rotation
    static constexpr uint32_t kAhead = 2;  // pieces on the GPU at once: one works, one waits behind it
    static constexpr uint32_t kChunk = 32; // packets a thread copies at a time
    uint32_t n, piece, pieces, chunks; // packets, packets per piece, pieces, chunks per piece
    std::function<void(uint32_t slot, uint32_t at, uint32_t first, uint32_t cnt)> in, out; // packets [first, +cnt) of the share, at `at` of the slot's batch
    std::function<int(uint32_t slot, uint32_t piece, uint32_t cnt)> submit;
    std::function<int(uint32_t slot)> poll;                                                // BNK_ETIMEDOUT: not yet
    std::atomic<uint32_t> in_next{0}, out_next{0}, gpu_done{0}, out_done{0};
    std::vector<std::atomic<uint32_t>> in_left, out_left;
    std::atomic<bool> stop{false};

    Share(uint32_t n_, uint32_t piece_)
        : n(n_), piece(piece_), pieces((n_ + piece_ - 1) / piece_), chunks((piece_ + kChunk - 1) / kChunk), in_left(pieces), out_left(pieces) {
        for (uint32_t p = 0; p < pieces; p++) {
            in_left[p].store(chunks, std::memory_order_relaxed);
            out_left[p].store(chunks, std::memory_order_relaxed);
        }
    }
    uint32_t Count(uint32_t p) const { return std::min(piece, n - p * piece); }
    void Chunk(uint32_t t, const std::function<void(uint32_t, uint32_t, uint32_t, uint32_t)> &f) const {
        const uint32_t p = t / chunks, at = t % chunks * kChunk, cnt = Count(p);
        if (at < cnt) f(p % kSlots, at, p * piece + at, std::min(kChunk, cnt - at));
    }
    // One copy, if there is one to do.
    bool Copy() {
        uint32_t t = out_next.load(std::memory_order_relaxed);
        if (t / chunks < gpu_done.load(std::memory_order_acquire) && t < pieces * chunks) {
            if (!out_next.compare_exchange_strong(t, t + 1, std::memory_order_acq_rel)) return true;
            Chunk(t, out);
            if (out_left[t / chunks].fetch_sub(1, std::memory_order_acq_rel) == 1) out_done.fetch_add(1, std::memory_order_release);
            return true;
        }
        t = in_next.load(std::memory_order_relaxed);
        if (t < pieces * chunks) {
            const uint32_t p = t / chunks;
            if (p >= kSlots && out_left[p - kSlots].load(std::memory_order_acquire) != 0) return false; // its ring is taken
            if (!in_next.compare_exchange_strong(t, t + 1, std::memory_order_acq_rel)) return true;
            Chunk(t, in);
            in_left[p].fetch_sub(1, std::memory_order_acq_rel);
            return true;
        }
        return false;
    }
    bool Over() const { return stop.load(std::memory_order_acquire) || out_done.load(std::memory_order_acquire) == pieces; }
    // The thread that drives the GPU; copies in between.  Returns the first error.
    int Drive() override {
        int rc = BNK_SUCCESS;
        uint32_t sent = 0, back = 0, idle = 0;
        while (!Over()) {
            if ((rc == BNK_SUCCESS || rc == BNK_EFULL) && sent < pieces && sent - back < kAhead && in_left[sent].load(std::memory_order_acquire) == 0) {
                const int r = submit(sent % kSlots, sent, Count(sent));
                sent++; // whatever was queued before an error has to be waited for as well
                if (r != BNK_SUCCESS) rc = r;
            }
            if (back < sent) { // BNK_EFULL (flows that found no place) is an outcome, the results are valid
                const int r = poll(back % kSlots);
                if (r != BNK_ETIMEDOUT) {
                    back++;
                    if (rc == BNK_SUCCESS || rc == BNK_EFULL) rc = r != BNK_SUCCESS ? r : rc;
                    if (rc == BNK_SUCCESS || rc == BNK_EFULL) gpu_done.store(back, std::memory_order_release);
                }
            } else if (rc != BNK_SUCCESS && rc != BNK_EFULL) {
                stop.store(true, std::memory_order_release);
            }
            Turn(idle);
        }
        return rc;
    }
    void Help() override {
        for (uint32_t idle = 0; !Over();) Turn(idle);
    }
    void Turn(uint32_t &idle) {
        if (Copy()) idle = 0;
        else if (++idle < 4000) Pause();
        else std::this_thread::yield(); // more threads than cores, or a GPU that is far behind
    }
};

// Threads that help with the copies of one GPU's shares.  They sleep between calls, after a moment of looking for the next.
class Crew {
  public:
    explicit Crew(uint32_t helpers) {
        try {
            threads_.reserve(helpers);
            for (uint32_t i = 0; i < helpers; i++) threads_.emplace_back([this] { Run(); });
        } catch (const std::exception &) { // as many as the process may have: a call's own thread does without them
        }
    }
    ~Crew() {
        {
            std::lock_guard<std::mutex> g(mu_);
            stop_.store(true);
        }
        cv_.notify_all();
        for (std::thread &t : threads_) t.join();
    }
    int Do(Task &t) {
        {
            std::lock_guard<std::mutex> g(mu_);
            task_ = &t;
            calls_.fetch_add(1);
        }
        cv_.notify_all();
        const int rc = t.Drive();
        {
            std::lock_guard<std::mutex> g(mu_);
            task_ = nullptr; // who has not come yet need not come
        }
        while (inside_.load(std::memory_order_acquire) != 0) Pause();
        return rc;
    }

  private:
    void Run() {
        uint64_t seen = 0;
        for (;;) {
            for (int i = 0; i < 1000 && calls_.load(std::memory_order_relaxed) == seen && !stop_.load(std::memory_order_relaxed); i++) Pause();
            Task *t;
            {
                std::unique_lock<std::mutex> g(mu_);
                cv_.wait(g, [&] { return stop_.load() || calls_.load() != seen; });
                if (stop_.load()) return;
                seen = calls_.load();
                t = task_;
                if (t) inside_.fetch_add(1, std::memory_order_acq_rel);
            }
            if (!t) continue;
            t->Help();
            inside_.fetch_sub(1, std::memory_order_acq_rel);
        }
    }
    std::mutex mu_;
    std::condition_variable cv_;
    Task *task_ = nullptr;
    std::atomic<uint64_t> calls_{0};
    std::atomic<bool> stop_{false};
    std::atomic<int> inside_{0};
    std::vector<std::thread> threads_;
};

} // namespace crew
