// memcpy split over the calling thread and a few workers (host_copy.cpp).
// No CUDA here: the tests compile this file alone, with threads of their own.
#pragma once
#include <atomic>
#include <condition_variable>
#include <cstddef>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace cpsgpu {

template <class Thread = std::thread> class CopyPool {
 public:
  // at most this many workers: a process at its thread limit has the ones
  // that could be started (an exception out of here would destroy running
  // threads and end the process)
  explicit CopyPool(int workers) {
    try {
      for (int k = 0; k < workers; k++) th_.emplace_back([this, k] { work(k); });
    } catch (const std::exception &) {
    }
  }
  ~CopyPool() {
    {
      std::lock_guard<std::mutex> lk(mu_);
      quit_ = true;
      gen_.fetch_add(1, std::memory_order_release);
    }
    cv_.notify_all();
    for (auto &t : th_) t.join();
  }
  void copy(void *dst, const void *src, size_t n) {
    const int parts = (int)th_.size() + 1;
    if (parts == 1 || n < (size_t(64) << 10)) {
      std::memcpy(dst, src, n);
      return;
    }
    dst_ = static_cast<char *>(dst);
    src_ = static_cast<const char *>(src);
    n_ = n;
    left_.store((int)th_.size(), std::memory_order_relaxed);
    {
      std::lock_guard<std::mutex> lk(mu_);
      gen_.fetch_add(1, std::memory_order_release);
    }
    cv_.notify_all();
    part((int)th_.size(), parts);
    // the workers' parts are as large as the one just done
    while (left_.load(std::memory_order_acquire) != 0) std::this_thread::yield();
  }

 private:
  void part(int k, int parts) {
    const size_t page = 4096, per = (n_ / parts + page - 1) / page * page, at = per * k;
    if (at >= n_) return;
    std::memcpy(dst_ + at, src_ + at, (k == parts - 1 || at + per > n_) ? n_ - at : per);
  }
  void work(int k) {
    unsigned seen = 0;
    for (;;) {
      // chunks of one transfer follow each other within microseconds: look
      // for the next one a while before sleeping
      for (int spin = 0; spin < 4000 && gen_.load(std::memory_order_acquire) == seen; spin++) std::this_thread::yield();
      if (gen_.load(std::memory_order_acquire) == seen) {
        std::unique_lock<std::mutex> lk(mu_);
        cv_.wait(lk, [&] { return gen_.load(std::memory_order_acquire) != seen; });
      }
      seen = gen_.load(std::memory_order_acquire);
      if (quit_) return;
      part(k, (int)th_.size() + 1);
      left_.fetch_sub(1, std::memory_order_release);
    }
  }
  std::vector<Thread> th_;
  std::mutex mu_;
  std::condition_variable cv_;
  std::atomic<unsigned> gen_{0};
  std::atomic<int> left_{0};
  bool quit_ = false;
  char *dst_ = nullptr;
  const char *src_ = nullptr;
  size_t n_ = 0;
};

}  // namespace cpsgpu
