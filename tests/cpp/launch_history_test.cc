// What a launch is told about the launches beside it (launch_history.h).
#include <cstdio>

#include "launch_history.h"

using fbgemm_b200::LaunchHistory;

#define EXPECT(GOT, WANT)                                                                            \
  do {                                                                                               \
    const long long got = (GOT), want = (WANT);                                                      \
    if (got != want) {                                                                               \
      std::printf("line %d: %s is %lld, not %lld\n", __LINE__, #GOT, got, want);                     \
      return 1;                                                                                      \
    }                                                                                                \
  } while (0)

int main() {
  char s[64];  // streams are addresses
  {
    LaunchHistory h;  // one stream: nothing beside it, ever
    for (int i = 0; i < 100; ++i) {
      EXPECT(h.launched(nullptr, 1000 + i), 0);
    }
    EXPECT(h.launched(&s[0], 5), 1099);  // (the default stream counts like any other)
  }
  {
    LaunchHistory h;  // two streams in turn: the other one's latest
    EXPECT(h.launched(&s[0], 10), 0);
    EXPECT(h.launched(&s[1], 20), 10);
    EXPECT(h.launched(&s[0], 11), 20);
    EXPECT(h.launched(&s[0], 12), 20);
    h.waited(&s[1]);
    EXPECT(h.launched(&s[0], 13), 0);
    h.waited(&s[0]);
    h.waited(&s[2]);
    EXPECT(h.launched(&s[1], 1), 0);
    for (int i = 0; i < LaunchHistory::kRecent - 1; ++i) {
      EXPECT(h.launched(&s[3], 7), 1);
    }
    EXPECT(h.launched(&s[3], 7), 0);  // long ago by now
  }
  {
    LaunchHistory h;  // as many streams as are remembered, and more
    for (int round = 0; round < 5; ++round) {
      for (int i = 0; i < LaunchHistory::kRecent; ++i) {
        EXPECT(h.launched(&s[i], 100), 100 * (round ? LaunchHistory::kRecent - 1 : i));
      }
    }
    for (int round = 0; round < 3; ++round) {
      for (int i = 0; i < 40; ++i) {
        EXPECT(h.launched(&s[20 + i], 100), 100 * (LaunchHistory::kRecent - 1));
      }
    }
  }
  return 0;
}
