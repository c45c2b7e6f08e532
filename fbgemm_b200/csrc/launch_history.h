// What runs beside a launch, as far as a context can tell.
//
// How many lanes share a bag, and how many registers a lane gets, is best chosen
// by the number of bags on the chip (pick_variant and launch_bags in
// bag_dispatch.cu), and small calls on several streams are on the chip together.
// A launch sees only itself; the context sees the streams of the launches before
// it.  The latest launch of every other stream among the last kRecent counts as
// running.  The choice has no influence on results.
#pragma once

#include <cstdint>
#include <mutex>

namespace fbgemm_b200 {

class LaunchHistory {
 public:
  static constexpr int kRecent = 16;

  // Notes a launch of `bags` bags on `stream`; returns the bags of the launches that count as running beside it.
  int64_t launched(const void* stream, int64_t bags) {
    std::lock_guard<std::mutex> lock(mu_);
    ++now_;
    int64_t beside = 0;
    int mine = 0;
    for (int i = 0; i < kRecent; ++i) {
      if (last_[i].at != 0 && last_[i].stream == stream) {
        last_[i].at = 0;
      } else if (last_[i].at != 0 && now_ - last_[i].at < kRecent) {
        beside += last_[i].bags;
      }
      mine = last_[i].at < last_[mine].at ? i : mine;  // the stream's own entry, else the oldest
    }
    last_[mine] = {stream, bags, now_};
    return beside;
  }

  // Everything on `stream` has completed.
  void waited(const void* stream) {
    std::lock_guard<std::mutex> lock(mu_);
    for (Launch& l : last_) {
      l.at = l.stream == stream ? 0 : l.at;
    }
  }

 private:
  struct Launch {
    const void* stream = nullptr;
    int64_t bags = 0;
    uint64_t at = 0;  // 0: none
  };
  std::mutex mu_;
  uint64_t now_ = 0;
  Launch last_[kRecent];
};

}  // namespace fbgemm_b200
