// See host_copy.h.  The helpers are shared by all contexts and calls of the
// process: at most kHelpers threads, started when a copy first wants them, and
// gone after a second without work.  A call that finds them busy with another
// call's copy copies alone.
#include "host_copy.h"

#if defined(__x86_64__)
#include <emmintrin.h>
#endif

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <thread>

#include <unistd.h>

namespace fbgemm_b200 {

namespace {

constexpr int kHelpers = 3;
constexpr size_t kWorthHelp = 512 * 1024;  // waking the helpers costs the copy of a few hundred KB
// Uploads go past the caches: the GPU alone reads the staging block, and its lines need not be fetched first (253 -> 218 us
// for the call of 10 000 bags in c_api.cu). So do results from this size on. Smaller ones are left in the caches for the
// caller, who reads them next; us for the call and a sum over its rows, past / through the caches:
// 64 KB 67 / 58, 256 KB 104 / 72, 512 KB 146 / 114, 1 MB 235 / 172, 2 MB 405 / 284; 5 MB 812 / 861, 10 MB 1480 / 1430 (the rows
// then come out of other cores' caches), 75 MB 11500 / 11600.
constexpr size_t kPastCaches = 4 << 20;
constexpr auto kIdle = std::chrono::seconds(1);
constexpr int kSpins = 2000;  // some 100 us without a slice to copy, then a helper sleeps

class Helpers {
 public:
  const pid_t pid = getpid();

  ~Helpers() {
    {
      std::lock_guard<std::mutex> l(mu_);
      stop_ = true;
    }
    wake_.notify_all();
    for (auto& t : threads_) {
      if (t.joinable()) {
        t.join();
      }
    }
  }

  bool copy(const CopySlice* slices, int count, int parts, bool ahead, const std::function<bool(int)>& ready,
            const std::function<bool(int)>& done) {
    // One copy at a time has the helpers.
    std::unique_lock<std::mutex> mine(in_use_, std::defer_lock);
    if (pid == getpid()) {
      (void)mine.try_lock();
    }
    size_t bytes = 0;
    for (int i = 0; i < count; ++i) {
      bytes += slices[i].bytes;
    }
    const bool past = ahead || bytes >= kPastCaches;
    struct Closing {  // however the copy ends, no helper holds a slice of it afterwards
      Helpers* helpers = nullptr;
      ~Closing() {
        if (helpers) {
          helpers->close();
        }
      }
    } closing;
    if (!ahead && pid == getpid() && bytes >= kWorthHelp) {
      alert();
    }
    bool ok = true;
    int end = 0;  // slices of the parts so far
    for (int p = 0; p < parts && ok; ++p) {
      if (!ahead && ready) {
        ok = ready(p);
        if (!ok) {
          break;
        }
      }
      // the helpers are not taken before there is something to copy
      if (p == 0 && mine.owns_lock() && bytes >= kWorthHelp && open(slices, count, ahead ? count : 0, past)) {
        closing.helpers = this;
      }
      const int begin = end;
      while (end < count && slices[end].part <= p) {
        ++end;
      }
      if (closing.helpers) {
        if (!ahead) {
          publish(end);
        }
        if (done) {
          while (left_[p].load(std::memory_order_acquire) > 0) {
            if (!claim_one()) {
              pause();
            }
          }
        }
      } else {
        for (int i = begin; i < end; ++i) {
          take(slices[i], past);
        }
      }
      ok = !done || done(p);
    }
    while (closing.helpers && claim_one()) {
    }
    return ok;
  }

 private:
  static void take(const CopySlice& s, bool past) {
    size_t done = 0;
#if defined(__x86_64__)
    if (past && reinterpret_cast<uintptr_t>(s.dst) % 16 == 0) {
      const __m128i* from = static_cast<const __m128i*>(s.src);
      __m128i* to = static_cast<__m128i*>(s.dst);
      for (; done + 64 <= s.bytes; done += 64, from += 4, to += 4) {
        const __m128i a = _mm_loadu_si128(from), b = _mm_loadu_si128(from + 1);
        const __m128i c = _mm_loadu_si128(from + 2), d = _mm_loadu_si128(from + 3);
        _mm_stream_si128(to, a);
        _mm_stream_si128(to + 1, b);
        _mm_stream_si128(to + 2, c);
        _mm_stream_si128(to + 3, d);
      }
      _mm_sfence();
    }
#endif
    std::memcpy(static_cast<char*>(s.dst) + done, static_cast<const char*>(s.src) + done, s.bytes - done);
  }

  static void pause() {
#if defined(__x86_64__)
    __builtin_ia32_pause();
#else
    std::this_thread::yield();
#endif
  }

  // Takes the next slice that is ready; false if there is none.
  bool claim_one() {
    int i = claimed_.load(std::memory_order_relaxed);
    while (i < ready_.load(std::memory_order_acquire)) {
      if (claimed_.compare_exchange_weak(i, i + 1, std::memory_order_acq_rel)) {
        take(slices_[i], past_);
        left_[slices_[i].part].fetch_sub(1, std::memory_order_acq_rel);
        return true;
      }
    }
    return false;
  }

  // Slices below `end` may be copied.  (Sequentially consistent, as work()'s counterpart is: either the sleeper is seen
  // here or it sees the new end.)
  void publish(int end) {
    ready_.store(end);
    if (sleeping_.load() > 0) {
      { std::lock_guard<std::mutex> l(mu_); }
      wake_.notify_all();
    }
  }

  // A copy is about to be opened: waking a helper takes as long as copying a megabyte, so they wake up while the first
  // rows are on their way (1 MB of rows 205 us without, 115 with), and do not keep other calls from being helped.
  void alert() {
    {
      std::lock_guard<std::mutex> l(mu_);
      if (stop_ || !start()) {
        return;
      }
      ++alerts_;
    }
    wake_.notify_all();
  }

  // Whether there are helpers: those that left for want of work are started again (mu_ held).
  bool start() {
    if (std::thread::hardware_concurrency() <= kHelpers + 1) {
      return false;
    }
    int have = 0;
    for (int i = 0; i < kHelpers; ++i) {
      if (threads_[i].joinable() && gone_[i]) {
        threads_[i].join();
      }
      if (!threads_[i].joinable()) {
        try {
          gone_[i] = false;
          threads_[i] = std::thread([this, i] { work(i); });
        } catch (...) {
          break;  // no thread to be had: fewer helpers, or the caller alone
        }
      }
      ++have;
    }
    return have > 0;
  }

  bool open(const CopySlice* slices, int count, int ready, bool past) {
    std::lock_guard<std::mutex> l(mu_);
    if (stop_ || !start()) {
      return false;
    }
    slices_ = slices;
    past_ = past;
    for (auto& l : left_) {
      l.store(0, std::memory_order_relaxed);
    }
    for (int i = 0; i < count; ++i) {
      left_[slices[i].part].fetch_add(1, std::memory_order_relaxed);
    }
    claimed_.store(0, std::memory_order_relaxed);
    ready_.store(ready, std::memory_order_release);
    open_.store(true, std::memory_order_release);
    wake_.notify_all();
    return true;
  }

  // No helper holds a slice of this copy after this returns.
  void close() {
    std::unique_lock<std::mutex> l(mu_);
    open_.store(false, std::memory_order_release);
    wake_.notify_all();
    done_.wait(l, [this] { return busy_ == 0; });
  }

  void work(int slot) {
    std::unique_lock<std::mutex> l(mu_);
    uint64_t seen = alerts_;
    while (true) {
      if (!wake_.wait_for(l, kIdle, [&] { return stop_ || open_.load(std::memory_order_acquire) || alerts_ != seen; })) {
        gone_[slot] = true;
        return;
      }
      if (stop_) {
        return;
      }
      if (!open_.load(std::memory_order_acquire)) {
        seen = alerts_;
        l.unlock();
        for (int i = 0; i < kSpins && !open_.load(std::memory_order_acquire); ++i) {
          pause();
        }
        l.lock();
        continue;
      }
      ++busy_;
      l.unlock();
      for (int idle = 0; open_.load(std::memory_order_acquire);) {
        if (claim_one()) {
          idle = 0;
        } else if (++idle < kSpins) {
          pause();
        } else {
          l.lock();
          sleeping_.fetch_add(1);
          wake_.wait(l, [this] { return !open_.load() || claimed_.load() < ready_.load(); });
          sleeping_.fetch_sub(1);
          l.unlock();
          idle = 0;
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
  std::thread threads_[kHelpers];
  bool gone_[kHelpers] = {};
  bool stop_ = false;
  int busy_ = 0;
  uint64_t alerts_ = 0;
  std::atomic<bool> open_{false};
  std::atomic<int> claimed_{0}, ready_{0}, sleeping_{0};
  std::atomic<int> left_[kCopyParts] = {};  // slices of each part that are not copied yet
  const CopySlice* slices_ = nullptr;
  bool past_ = false;
};

}  // namespace

bool copy_slices(const CopySlice* slices, int count, int parts, bool ahead, const std::function<bool(int)>& ready,
                 const std::function<bool(int)>& done) {
  // A forked child has neither the threads nor a use for the locks: it copies alone, and does not wait for threads that
  // are not there when it exits.
  struct Owner {
    Helpers* helpers = new Helpers;
    ~Owner() {
      if (helpers->pid == getpid()) {
        delete helpers;
      }
    }
  };
  static Owner owner;
  return owner.helpers->copy(slices, count, parts, ahead, ready, done);
}

}  // namespace fbgemm_b200
