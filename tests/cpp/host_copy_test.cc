// The threaded host copies by themselves: host_copy_test exact | fork | idle | again
#include <sys/resource.h>
#include <sys/wait.h>
#include <signal.h>
#include <unistd.h>

#include <algorithm>
#include <chrono>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <stdexcept>
#include <string>
#include <thread>
#include <vector>

#include "host_copy.h"

using fbgemm_b200::copy_slices;
using fbgemm_b200::CopySlice;

namespace {

struct Copy {
  std::vector<uint8_t> src, dst;
  std::vector<CopySlice> slices;
  Copy(size_t bytes, size_t slice, int parts, size_t skew) : src(bytes + skew), dst(bytes + 2 * skew, 0) {
    for (size_t i = 0; i < src.size(); ++i) {
      src[i] = (uint8_t)(i * 2654435761u >> 11);
    }
    for (size_t at = 0; at < bytes; at += slice) {
      const int part = (int)(at * parts / bytes);
      slices.push_back({dst.data() + skew + at, src.data() + skew + at, std::min(slice, bytes - at), part});
    }
  }
  bool same(size_t skew, size_t upto) const {
    return std::memcmp(dst.data() + skew, src.data() + skew, upto) == 0;
  }
};

int exact() {
  for (size_t bytes : {size_t(1), size_t(1000), size_t(600 * 1024 + 7), size_t(5 << 20)}) {
    for (int parts : {1, 3, 8}) {
      for (size_t skew : {size_t(0), size_t(1)}) {
        for (bool ahead : {false, true}) {
          Copy c(bytes, 100 * 1024, parts, skew);
          int readied = 0, finished = 0;
          const bool ok = copy_slices(
              c.slices.data(), (int)c.slices.size(), parts, ahead, [&](int p) { return p == readied++; },
              [&](int p) { return p == finished++; });
          if (!ok || finished != parts || readied != (ahead ? 0 : parts) || !c.same(skew, bytes)) {
            std::printf("bytes %zu parts %d skew %zu ahead %d\n", bytes, parts, skew, ahead);
            return 1;
          }
        }
      }
    }
  }
  Copy c(4 << 20, 64 * 1024, 4, 0);   // ended early, with an error and with an exception; the next copy is whole again
  if (copy_slices(c.slices.data(), (int)c.slices.size(), 4, false, [](int p) { return p < 2; }, nullptr)) {
    return 2;
  }
  bool thrown = false;
  try {
    copy_slices(c.slices.data(), (int)c.slices.size(), 4, true, nullptr,
                [](int p) -> bool { return p < 1 ? true : throw std::runtime_error("part 1"); });
  } catch (const std::runtime_error&) {
    thrown = true;
  }
  Copy d(4 << 20, 64 * 1024, 4, 0);
  return thrown && copy_slices(d.slices.data(), (int)d.slices.size(), 4, false, nullptr, nullptr) && d.same(0, 4 << 20) ? 0 : 3;
}

// A child of a process whose helpers live copies, and ends by exit().
int forked() {
  Copy c(4 << 20, 64 * 1024, 1, 0);
  copy_slices(c.slices.data(), (int)c.slices.size(), 1, true, nullptr, nullptr);
  const pid_t child = fork();
  if (child == 0) {
    Copy d(4 << 20, 64 * 1024, 1, 0);
    copy_slices(d.slices.data(), (int)d.slices.size(), 1, true, nullptr, nullptr);
    std::exit(d.same(0, 4 << 20) ? 0 : 1);
  }
  for (int i = 0; i < 100; ++i) {
    int status = 0;
    if (waitpid(child, &status, WNOHANG) == child) {
      return WIFEXITED(status) ? WEXITSTATUS(status) : 2;
    }
    std::this_thread::sleep_for(std::chrono::milliseconds(100));
  }
  kill(child, SIGKILL);
  waitpid(child, nullptr, 0);
  std::printf("the child did not end\n");
  return 3;
}

double cpu_seconds() {
  rusage u;
  getrusage(RUSAGE_SELF, &u);
  return (double)(u.ru_utime.tv_sec + u.ru_stime.tv_sec) + 1e-6 * (double)(u.ru_utime.tv_usec + u.ru_stime.tv_usec);
}

// Waiting for parts to arrive keeps no core busy, neither for the first nor for the later ones.
int idle() {
  Copy c(4 << 20, 64 * 1024, 3, 0);
  copy_slices(c.slices.data(), (int)c.slices.size(), 3, false, nullptr, nullptr);  // the helpers are there
  for (int slow = 0; slow < 3; ++slow) {
    const double before = cpu_seconds();
    copy_slices(
        c.slices.data(), (int)c.slices.size(), 3, false,
        [&](int p) {
          if (p == slow) {
            std::this_thread::sleep_for(std::chrono::milliseconds(400));
          }
          return true;
        },
        nullptr);
    const double used = cpu_seconds() - before;
    if (used > 0.1) {
      std::printf("%.3f s of processor time while part %d was waited for\n", used, slow);
      return 1;
    }
  }
  return c.same(0, 4 << 20) ? 0 : 2;
}

// Copies after the helpers have left for want of work.
int again() {
  for (int i = 0; i < 2; ++i) {
    Copy c(4 << 20, 64 * 1024, 1, 0);
    if (!copy_slices(c.slices.data(), (int)c.slices.size(), 1, true, nullptr, nullptr) || !c.same(0, 4 << 20)) {
      return 1;
    }
    std::this_thread::sleep_for(std::chrono::milliseconds(1500));
  }
  return 0;
}

}  // namespace

int main(int argc, char** argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  return what == "exact" ? exact() : what == "fork" ? forked() : what == "idle" ? idle() : what == "again" ? again() : 64;
}
