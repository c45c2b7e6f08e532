// Which lookups of a handful of bags go to a block per bag (few_bags_rule.h), on 148 SMs.
#include <cstdio>

#include "few_bags_rule.h"

using fbgemm_b200::FewBagsCall;
using fbgemm_b200::few_bags_pay;

#define EXPECT(GOT, WANT)                                                                            \
  do {                                                                                               \
    const long long got = (GOT), want = (WANT);                                                      \
    if (got != want) {                                                                               \
      std::printf("line %d: %s is %lld, not %lld\n", __LINE__, #GOT, got, want);                     \
      return 1;                                                                                      \
    }                                                                                                \
  } while (0)

int main() {
  // rows of words: `average` rows a bag, `bags` bags of 128 columns a tile
  const auto words = [](int bits, int64_t tiles, int64_t bags, int64_t average, int64_t beside = 0) {
    return few_bags_pay({bits, true, 0, 1, false, tiles, bags, beside, bags * average}, 148);
  };
  // rows of halves or bytes
  const auto units = [](int n, int chunks, int64_t tiles, int64_t bags, int64_t average, bool mapped = false) {
    return few_bags_pay({8, false, n, chunks, mapped, tiles, bags, 0, bags * average}, 148);
  };
  // short bags of 8- and 4-bit rows in one tile: a warp's one stretch is faster
  const int64_t few[] = {1, 10, 100, 250};
  for (int64_t bags : few) {
    EXPECT(words(8, 1, bags, 4), 0);
    EXPECT(words(8, 1, bags, 16), 0);
    EXPECT(words(8, 1, bags, 31), 0);
    EXPECT(words(8, 1, bags, 32), 1);
    EXPECT(words(8, 1, bags, 100), 1);
    EXPECT(words(4, 1, bags, 16), 0);
    EXPECT(words(4, 1, bags, 20), 1);
    EXPECT(words(2, 1, bags, 4), 1);
  }
  EXPECT(words(8, 2, 100, 4), 1);
  // so many blocks an SM
  EXPECT(words(8, 1, 592, 32), 1);
  EXPECT(words(8, 1, 593, 32), 0);
  EXPECT(words(8, 1, 592, 32, 1), 0);
  EXPECT(words(8, 1, 1184, 59), 0);
  EXPECT(words(8, 1, 1184, 60), 1);
  EXPECT(words(8, 1, 1185, 60), 0);
  EXPECT(words(4, 1, 296, 20), 1);
  EXPECT(words(4, 1, 297, 20), 0);
  EXPECT(words(8, 2, 148, 4), 1);
  EXPECT(words(8, 2, 149, 4), 0);
  EXPECT(words(8, 2, 296, 20), 1);
  EXPECT(words(8, 2, 297, 59), 0);
  EXPECT(words(8, 2, 444, 60), 1);
  EXPECT(words(8, 2, 445, 60), 0);
  EXPECT(words(8, 2, 592, 90), 1);
  EXPECT(words(8, 2, 593, 100), 0);
  EXPECT(words(2, 2, 296, 4), 1);
  EXPECT(words(2, 2, 592, 60), 1);
  // halves and bytes
  EXPECT(units(43, 1, 1, 100, 16), 0);
  EXPECT(units(43, 1, 1, 100, 20), 1);
  EXPECT(units(43, 1, 1, 590, 20), 0);
  EXPECT(units(43, 1, 1, 590, 30), 1);
  EXPECT(units(64, 2, 2, 100, 20), 1);
  EXPECT(units(128, 2, 2, 100, 30), 0);
  EXPECT(units(128, 2, 2, 100, 60), 1);
  EXPECT(units(128, 2, 2, 250, 60), 0);
  EXPECT(units(101, 4, 1, 100, 15), 0);
  EXPECT(units(101, 4, 1, 590, 16), 1);
  // behind a pruning map
  const auto mapped = [](int bits, int64_t tiles, int64_t bags, int64_t average) {
    return few_bags_pay({bits, true, 0, 1, true, tiles, bags, 0, bags * average}, 148);
  };
  EXPECT(mapped(8, 1, 10, 39), 0);
  EXPECT(mapped(8, 1, 10, 40), 1);
  EXPECT(mapped(8, 2, 10, 5), 0);
  EXPECT(mapped(8, 2, 296, 40), 1);
  EXPECT(mapped(8, 2, 297, 100), 0);
  EXPECT(mapped(4, 1, 10, 31), 0);
  EXPECT(mapped(4, 1, 296, 32), 1);
  EXPECT(mapped(4, 1, 297, 55), 0);
  EXPECT(mapped(4, 1, 592, 56), 1);
  EXPECT(mapped(4, 1, 593, 100), 0);
  EXPECT(mapped(2, 1, 10, 19), 0);
  EXPECT(mapped(2, 1, 10, 20), 1);
  EXPECT(units(43, 1, 1, 100, 31, true), 0);
  EXPECT(units(43, 1, 1, 100, 32, true), 1);
  EXPECT(units(128, 2, 2, 10, 100, true), 0);
  EXPECT(units(101, 4, 1, 590, 16, true), 1);
  // no bags, no rows, and numbers whose products need 64 bits
  EXPECT(words(8, 1, 0, 100), 0);
  EXPECT(words(8, 1, 10, 0), 0);
  EXPECT(words(8, 1, 0x7fffffffffLL, 100), 0);
  EXPECT(few_bags_pay({8, true, 0, 1, false, 1 << 20, 1LL << 40, 1LL << 40, 0x7fffff00LL}, 148), 0);
  return 0;
}
