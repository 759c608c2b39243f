// Worker threads that an engine or batch keeps for its host-side output work
// (widening byte rows, faulting in the pages of fresh output buffers).
// Creating 16 threads takes 0.7-0.9 ms on the GPU host, more than the work of
// most calls. One job runs at a time; the owner serialises its calls.
#pragma once

#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstddef>
#include <cstdint>
#include <exception>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

#include "host_graph.h"

namespace msbfs {

class HostPool {
 public:
  HostPool() = default;
  HostPool(const HostPool&) = delete;
  HostPool& operator=(const HostPool&) = delete;
  ~HostPool() {
    wait();
    {
      std::lock_guard<std::mutex> lk(mu_);
      stop_ = true;
      job_.fetch_add(1);
    }
    cv_.notify_all();
    for (std::thread& t : threads_) t.join();
  }
  // Creates threads up to n (at most max_workers()) and returns how many of n
  // there are: fewer when the system gives no more. Waits for the job before.
  unsigned reserve(unsigned n) {
    wait();
    try {
      while (threads_.size() < n) {
        const unsigned k = (unsigned)threads_.size();
        threads_.emplace_back([this, k, seen = job_.load()] { work(k, seen); });
      }
    } catch (const std::exception&) {  // callers are C entry points
    }
    return std::min(n, (unsigned)threads_.size());
  }
  // Starts body(k) for every k < n on a thread each, and returns. Shares that no
  // thread can be had for run here, before the return.
  void start(unsigned n, std::function<void(unsigned)> body) {
    const unsigned have = reserve(n);
    {
      std::lock_guard<std::mutex> lk(mu_);  // a worker takes job and share together
      body_ = std::move(body);
      active_ = have;
      left_.store(have);
      job_.fetch_add(1);
    }
    cv_.notify_all();
    for (unsigned k = have; k < n; ++k) body_(k);
  }
  void wait() {
    if (left_.load(std::memory_order_acquire) == 0) return;
    std::unique_lock<std::mutex> lk(mu_);
    done_.wait(lk, [this] { return left_.load() == 0; });
  }
  static unsigned max_workers() { return (unsigned)host_threads(); }

 private:
  void work(unsigned k, uint64_t seen) {
    for (;;) {
      // A short spin first: the next of a row of small jobs (one per result
      // array) then starts without a sleep and a wake-up.
      const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(40);
      while (job_.load(std::memory_order_acquire) == seen && std::chrono::steady_clock::now() < until)
        std::this_thread::yield();
      unsigned n;
      {
        std::unique_lock<std::mutex> lk(mu_);
        cv_.wait(lk, [&] { return job_.load() != seen; });
        if (stop_) return;
        seen = job_.load();
        n = active_;
      }
      if (k >= n) continue;
      body_(k);
      if (left_.fetch_sub(1) == 1) {
        std::lock_guard<std::mutex> lk(mu_);
        done_.notify_all();
      }
    }
  }
  std::vector<std::thread> threads_;
  std::function<void(unsigned)> body_;
  std::mutex mu_;
  std::condition_variable cv_, done_;
  std::atomic<uint64_t> job_{0};
  std::atomic<unsigned> left_{0};
  unsigned active_ = 0;  // workers of the running job
  bool stop_ = false;
};

// Starts making the pages inside [p, p + bytes) present, without touching what
// they hold (pool.wait() when that must be done). A device-to-host copy into
// untouched pageable memory faults them in one after the other, at 27 GB/s
// against 180 once they are present; 4 threads fault at 84. Where the
// kernel does not know the request the pages stay as they are.
inline void prefault(HostPool& pool, void* p, size_t bytes) {
#ifdef MADV_POPULATE_WRITE
  constexpr int POPULATE = MADV_POPULATE_WRITE;
#else
  constexpr int POPULATE = 23;
#endif
  constexpr unsigned FAULTERS = 4;  // 351 MB: 10.7 / 6.0 / 4.2 / 6.5 / 6.0 ms with 1 / 2 / 4 / 8 / 16
  // Shares begin on 2 MB boundaries: a transparent huge page is one fault.
  constexpr uintptr_t HUGE = uintptr_t(2) << 20;
  const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
  const uintptr_t lo = ((uintptr_t)p + page - 1) / page * page;
  const uintptr_t hi = ((uintptr_t)p + bytes) / page * page;
  if (hi <= lo || bytes < HUGE) return;
  const uintptr_t first = lo / HUGE, pieces = (hi - 1) / HUGE - first + 1;
  const unsigned n = (unsigned)std::min<uintptr_t>(std::min(HostPool::max_workers(), FAULTERS), pieces);
  pool.start(n, [=](unsigned k) {
    const uintptr_t b = std::max(lo, (first + pieces * k / n) * HUGE);
    const uintptr_t e = std::min(hi, (first + pieces * (k + 1) / n) * HUGE);
    if (b < e) (void)madvise(reinterpret_cast<void*>(b), e - b, POPULATE);
  });
}

}  // namespace msbfs
