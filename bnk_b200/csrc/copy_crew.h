// Copies between callers' buffers and the pinned ring of a queue, shared with helper threads.  One thread copies full-size
// packets at ~13 GB/s (each packet's lines come from memory or from another core's cache), which is what bounds a caller
// that hands in one upstream batch after the other: eight calls of 128 x 1420 B each way through the queues 495 us, of
// them ~320 copying, with two helpers 380; 14 of 200 x 600 B 845 and 510.
//
// Helpers are for that caller only.  They are woken when copies follow one another closely and go back to sleep when
// none has come for a while; a lone batch now and then never wakes them.  Where several threads copy at the same time
// they are the parallelism themselves, and everybody copies alone.
#pragma once

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

class CopyCrew {
  public:
    explicit CopyCrew(uint32_t helpers) {
        try {
            threads_.reserve(helpers);
            for (uint32_t i = 0; i < helpers; i++) threads_.emplace_back([this] { help(); });
        } catch (const std::exception &) { // as many as the process may have
        }
    }
    ~CopyCrew() {
        {
            std::lock_guard<std::mutex> g(mu_);
            stop_.store(true, std::memory_order_relaxed);
        }
        cv_.notify_all();
        for (std::thread &t : threads_) t.join();
    }
    CopyCrew(const CopyCrew &) = delete;
    // A quarter of the cores at most, two at most: with four the two measurements above are 350 and 545 us.
    static uint32_t helpers_for(uint32_t cores) { return std::min(2u, cores / 4); }

    // Calls part(0) .. part(n - 1), each once, in any order and on any thread, and returns when all have returned.
    template <typename Part>
    void run(uint32_t n, Part part) {
        if (n > 1 && !threads_.empty()) {
            const int64_t now = clock_ns();
            if (busy_.exchange(true, std::memory_order_acquire)) {
                crowded_.store(now, std::memory_order_relaxed);
            } else {
                const bool shared = now - crowded_.load(std::memory_order_relaxed) > kCrowdedNs && helpers_awake(now);
                if (shared) {
                    call_ = [](void *p, uint32_t i) { (*static_cast<Part *>(p))(i); };
                    arg_ = &part;
                    done_.store(0, std::memory_order_relaxed);
                    const uint64_t gen = (work_.load(std::memory_order_relaxed) >> 32) + 1;
                    work_.store(gen << 32 | (uint64_t)n << 16, std::memory_order_release);
                    while (take()) {}
                    for (uint32_t spins = 1; done_.load(std::memory_order_acquire) != n; spins++) {
                        if (spins & 0xfffu) relax();
                        else std::this_thread::yield(); // a helper has lost its core
                    }
                } else {
                    for (uint32_t i = 0; i < n; i++) part(i);
                }
                last_ = clock_ns();
                busy_.store(false, std::memory_order_release);
                return;
            }
        }
        for (uint32_t i = 0; i < n; i++) part(i);
    }

  private:
    static constexpr int64_t kCloseNs = 30'000;     // copies this close together are one caller's burst
    static constexpr int64_t kStayNs = 60'000;      // a helper stays awake this long without work
    static constexpr int64_t kCrowdedNs = 1'000'000; // how long several threads copying at once are remembered

    static int64_t clock_ns() { return std::chrono::steady_clock::now().time_since_epoch().count(); }
    static void relax() {
#if defined(__x86_64__) || defined(__i386__)
        __builtin_ia32_pause();
#else
        std::this_thread::yield();
#endif
    }
    // Is a helper there?  Wakes them when this copy follows the last one closely.
    bool helpers_awake(int64_t now) {
        if (awake_.load(std::memory_order_relaxed) != 0) return true;
        if (now - last_ > kCloseNs) return false;
        {
            std::lock_guard<std::mutex> g(mu_);
            wake_++;
        }
        cv_.notify_all();
        return true;
    }
    // One part of the work at hand, if one is left.  work_: number of the work, its parts, the next part.  Who moves the last
    // field on holds that part, and the caller does not return, or change call_ and arg_, before it is done.
    bool take() {
        uint64_t w = work_.load(std::memory_order_acquire);
        while ((w & 0xffff) < (w >> 16 & 0xffff)) {
            if (!work_.compare_exchange_weak(w, w + 1, std::memory_order_acq_rel, std::memory_order_acquire)) continue;
            call_(arg_, (uint32_t)(w & 0xffff));
            done_.fetch_add(1, std::memory_order_release);
            return true;
        }
        return false;
    }
    void help() {
        uint64_t seen = 0;
        for (;;) {
            {
                std::unique_lock<std::mutex> g(mu_);
                cv_.wait(g, [&] { return stop_.load(std::memory_order_relaxed) || wake_ != seen; });
                if (stop_.load(std::memory_order_relaxed)) return;
                seen = wake_;
                awake_.fetch_add(1, std::memory_order_relaxed);
            }
            for (int64_t until = clock_ns() + kStayNs; !stop_.load(std::memory_order_relaxed) && clock_ns() < until;) {
                for (int i = 0; i < 64; i++) {
                    if (take()) until = clock_ns() + kStayNs;
                    else relax();
                }
            }
            awake_.fetch_sub(1, std::memory_order_relaxed);
        }
    }
    std::atomic<uint64_t> work_{0};
    void (*call_)(void *, uint32_t) = nullptr;
    void *arg_ = nullptr;
    alignas(64) std::atomic<uint32_t> done_{0};
    alignas(64) std::atomic<bool> busy_{false};
    std::atomic<int64_t> crowded_{INT64_MIN / 2};
    int64_t last_ = INT64_MIN / 2; // end of the last copy (whoever holds busy_)
    std::atomic<uint32_t> awake_{0};
    std::atomic<bool> stop_{false};
    std::mutex mu_;
    std::condition_variable cv_;
    uint64_t wake_ = 0; // under mu_
    std::vector<std::thread> threads_; // last: they use the rest
};
