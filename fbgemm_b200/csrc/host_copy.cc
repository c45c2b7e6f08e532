// See host_copy.h.  The helpers are shared by all contexts and calls of the
// process: at most kHelpers threads, started when a copy first wants them, and
// gone after a second without work.  A call that finds them busy with another
// call's copy copies alone.
#include "host_copy.h"

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

namespace fbgemm_b200 {

namespace {

constexpr int kHelpers = 3;
constexpr auto kIdle = std::chrono::seconds(1);

class Helpers {
 public:
  ~Helpers() {
    {
      std::lock_guard<std::mutex> l(mu_);
      stop_ = true;
    }
    wake_.notify_all();
    for (auto& t : threads_) {
      t.join();
    }
  }

  bool copy(const CopySlice* slices, int count, const std::function<bool(int)>& ready) {
    // One copy at a time has the helpers.
    std::unique_lock<std::mutex> mine(in_use_, std::try_to_lock);
    const bool helped = mine.owns_lock() && count > 1 && open(slices, count);
    bool ok = true;
    int next = 0;  // without helpers
    for (int i = 0; i < count; ++i) {
      ok = ready(i);
      if (!ok) {
        break;
      }
      if (helped) {
        ready_.store(i + 1, std::memory_order_release);
      } else {
        take(slices[next++]);
      }
    }
    if (helped) {
      while (claim_one()) {
      }
      close();
    }
    return ok;
  }

 private:
  static void take(const CopySlice& s) { std::memcpy(s.dst, s.src, s.bytes); }

  // Takes the next slice that is ready; false if there is none.
  bool claim_one() {
    int i = claimed_.load(std::memory_order_relaxed);
    while (i < ready_.load(std::memory_order_acquire)) {
      if (claimed_.compare_exchange_weak(i, i + 1, std::memory_order_acq_rel)) {
        take(slices_[i]);
        return true;
      }
    }
    return false;
  }

  bool open(const CopySlice* slices, int count) {
    std::lock_guard<std::mutex> l(mu_);
    if (stop_) {
      return false;
    }
    reap();
    const unsigned cores = std::thread::hardware_concurrency();
    const int want = cores > kHelpers + 1 ? kHelpers : 0;
    while ((int)threads_.size() < want) {
      try {
        const size_t slot = threads_.size();
        gone_[slot] = false;
        threads_.emplace_back([this, slot] { work(slot); });
      } catch (...) {
        break;  // no thread to be had: the callers copy
      }
    }
    if (threads_.empty()) {
      return false;
    }
    slices_ = slices;
    (void)count;
    claimed_.store(0, std::memory_order_relaxed);
    ready_.store(0, std::memory_order_relaxed);
    open_.store(true, std::memory_order_release);
    wake_.notify_all();
    return true;
  }

  // No helper holds a slice of this copy after this returns.
  void close() {
    std::unique_lock<std::mutex> l(mu_);
    open_.store(false, std::memory_order_release);
    done_.wait(l, [this] { return busy_ == 0; });
  }

  // Threads that left for want of work (mu_ held).
  void reap() {
    for (size_t i = 0; i < threads_.size(); ++i) {
      if (!gone_[i]) {
        return;  // they leave together or not at all worth restarting one by one
      }
    }
    for (auto& t : threads_) {
      t.join();
    }
    threads_.clear();
  }

  void work(size_t slot) {
    std::unique_lock<std::mutex> l(mu_);
    while (true) {
      if (!wake_.wait_for(l, kIdle, [this] { return stop_ || open_.load(std::memory_order_acquire); })) {
        gone_[slot] = true;
        return;
      }
      if (stop_) {
        return;
      }
      ++busy_;
      l.unlock();
      while (open_.load(std::memory_order_acquire)) {
        if (!claim_one()) {
#if defined(__x86_64__)
          __builtin_ia32_pause();
#else
          std::this_thread::yield();
#endif
        }
      }
      l.lock();
      if (--busy_ == 0) {
        done_.notify_all();
      }
    }
  }

  std::mutex in_use_;
  std::mutex mu_;
  std::condition_variable wake_, done_;
  std::vector<std::thread> threads_;
  bool gone_[kHelpers] = {};
  bool stop_ = false;
  int busy_ = 0;
  std::atomic<bool> open_{false};
  std::atomic<int> claimed_{0}, ready_{0};
  const CopySlice* slices_ = nullptr;
};

}  // namespace

bool copy_slices(const CopySlice* slices, int count, const std::function<bool(int)>& ready) {
  static Helpers helpers;
  return helpers.copy(slices, count, ready);
}

}  // namespace fbgemm_b200
