// memcpy split over the calling thread and a few workers (host_copy.cpp).
// No CUDA here: the tests compile this file alone, with threads of their own.
//
// A copy is cut into blocks which the caller and the workers claim one by
// one, so the caller never waits for a worker that is not running, only for
// blocks that a worker has begun.  That matters because the caller's own
// threads may hold the cores: OpenBLAS's spin for ~0.1 s after a threaded
// call, libgomp's after a parallel loop.  With a fixed part per worker and a
// wait for all of them (the earlier form) every chunk then took a scheduler
// slice: RHMC force 7.4 ms, right after a numpy dot product 99 ms.
#pragma once
#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstddef>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace cpsgpu {

// One thread at a time calls copy(), crowded() (host_copy.cpp's lock).
template <class Thread = std::thread> class CopyPool {
  using clk = std::chrono::steady_clock;
  // 16 / 32 / 64 KiB: MatPcDagMatPc, DWF 8^4 Ls=8 0.269 / 0.273 / 0.314 ms,
  // RHMC force, DWF 16^4 Ls=8 7.1 / 7.2 / 7.4 ms
  static constexpr size_t BLOCK = size_t(16) << 10;
  // A worker looks this long for the next copy before it sleeps: longer than
  // the pause between the chunks of a transfer.  300 us as fast as 2 ms; 50 us:
  // force 9.3 ms
  static constexpr auto LINGER = std::chrono::microseconds(300);
  // a block takes a few us: a caller that waits this long for one has met a
  // worker that lost its core in the middle
  static constexpr auto STALL = std::chrono::microseconds(500);
  static constexpr auto SHORTEST = std::chrono::milliseconds(50), LONGEST = std::chrono::milliseconds(1600);

 public:
  // at most this many workers: a process at its thread limit has the ones
  // that could be started (an exception out of here would destroy running
  // threads and end the process)
  explicit CopyPool(int workers) {
    try {
      for (int k = 0; k < workers; k++) th_.emplace_back([this] { work(); });
    } catch (const std::exception &) {
    }
  }
  ~CopyPool() {
    {
      std::lock_guard<std::mutex> lk(mu_);
      quit_ = true;
    }
    cv_.notify_all();
    for (auto &t : th_) t.join();
  }
  int workers() const { return (int)th_.size(); }
  // a worker lost its core lately: for a while the caller is better off
  // without the workers (50 ms, twice as long each time it happens again
  // within the time after that, at most 1.6 s)
  bool crowded() const { return clk::now() < alone_until_; }
  void copy(void *dst, const void *src, size_t n) {
    const unsigned blocks = (unsigned)((n + BLOCK - 1) / BLOCK);
    if (th_.empty() || blocks < 2 || crowded()) {
      std::memcpy(dst, src, n);
      return;
    }
    dst_ = static_cast<char *>(dst);
    src_ = static_cast<const char *>(src);
    n_ = n;
    done_.store(0, std::memory_order_relaxed);
    left_.store(blocks);  // publishes the above to whoever claims a block
    // (left_ and sleepers_ in the one total order: either the worker going to
    // sleep sees the blocks or this thread sees the sleeper)
    if (sleepers_.load() > 0) {
      { std::lock_guard<std::mutex> lk(mu_); }
      cv_.notify_one();  // who wakes the others
    }
    unsigned mine = 0, k;
    while (claim(k)) {
      block(k);
      mine++;
    }
    const unsigned theirs = blocks - mine;
    if (done_.load(std::memory_order_acquire) == theirs) return;
    const clk::time_point t0 = clk::now();
    while (done_.load(std::memory_order_acquire) != theirs) std::this_thread::yield();
    const clk::time_point t1 = clk::now();
    if (t1 - t0 > STALL) {
      alone_ = t1 < alone_until_ + alone_ ? std::min<clk::duration>(2 * alone_, LONGEST) : clk::duration(SHORTEST);
      alone_until_ = t1 + alone_;
    }
  }

 private:
  // the blocks not yet claimed are 0 .. left_ - 1; a copy ends only after its
  // last claimed block, so what a claim reads is of the copy it belongs to
  bool claim(unsigned &k) {
    unsigned v = left_.load(std::memory_order_acquire);
    while (v)
      if (left_.compare_exchange_weak(v, v - 1, std::memory_order_acq_rel, std::memory_order_acquire)) {
        k = v - 1;
        return true;
      }
    return false;
  }
  void block(unsigned k) {
    const size_t at = BLOCK * k;
    std::memcpy(dst_ + at, src_ + at, n_ - at < BLOCK ? n_ - at : BLOCK);
  }
  void work() {
    for (;;) {
      unsigned k;
      while (claim(k)) {
        block(k);
        done_.fetch_add(1, std::memory_order_release);
      }
      const clk::time_point until = clk::now() + LINGER;
      bool more = false;
      do {
        for (int s = 0; s < 16 && !(more = left_.load(std::memory_order_relaxed) != 0); s++) std::this_thread::yield();
      } while (!more && clk::now() < until);
      if (more) continue;
      {
        std::unique_lock<std::mutex> lk(mu_);
        sleepers_.fetch_add(1);
        cv_.wait(lk, [&] { return left_.load() != 0 || quit_; });
        sleepers_.fetch_sub(1);
        if (quit_) return;
      }
      if (sleepers_.load() > 0) cv_.notify_all();
    }
  }
  std::vector<Thread> th_;
  std::mutex mu_;
  std::condition_variable cv_;
  std::atomic<unsigned> left_{0}, done_{0};
  std::atomic<int> sleepers_{0};
  bool quit_ = false;
  char *dst_ = nullptr;
  const char *src_ = nullptr;
  size_t n_ = 0;
  clk::time_point alone_until_{};
  clk::duration alone_{};
};

}  // namespace cpsgpu
