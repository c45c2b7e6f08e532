// When a lookup in one quantized table is one of a handful of bags, for which a
// block per bag and 128 columns (few_bags_kernel.cu) is faster than a warp per
// bag and tile (bag_kernel.cuh).  The choice has no influence on results.
//
// A warp resolves 32 rows at a time and adds them up from registers, 12 in
// flight: up to 32 rows a bag its chain is no longer than the block's, which
// copies rows through shared memory and has barriers besides.  Every further
// stretch of 32 is a chain of its own, where the block has 256 rows on the way.
// Only the average length of the bags is known here.  us per call by warps / by
// blocks, enqueued calls one behind the other, 100 bags (b250, b590: as many)
// of lengths that are all the same / even between 1 and twice the average:
//                  16 rows                20 rows                30 rows                64 rows (even)
//   8-bit D = 64   2.87/3.24  3.23/3.88   3.01/3.54  4.08/4.07   3.44/4.11  4.64/4.14   8.93/4.74  b590 9.22/7.27
//   8-bit D = 128  2.90/3.26  3.31/3.98   3.00/3.49  4.08/4.09   3.40/4.07  4.68/4.24   9.49/4.77  b590 9.79/7.04
//   4-bit D = 128  2.87/2.97  3.30/3.42   2.97/3.11  4.04/3.51   3.37/3.44  4.69/3.64   9.37/4.26  b590 9.73/7.33
//   2-bit D = 128  2.87/2.63  3.30/2.95   2.96/2.80  4.10/3.04   3.40/3.06  4.64/3.10
//   8-bit D = 256  3.28/3.28  4.14/4.08   3.55/3.50  5.17/4.22   4.24/4.17  6.19/4.31   10.7/5.3   b590 11.1/11.6
//   4-bit D = 256  2.98/2.91  3.69/3.48   3.27/3.19  4.65/3.63   3.78/3.52  5.40/3.73   9.59/4.55  b590 9.85/9.57
//   8-bit D = 86   3.35/3.64  3.89/3.87   3.48/3.81  4.98/4.09   4.10/4.15  5.96/4.58   10.6/6.9   b590 10.8/8.8
//   8-bit D = 150  3.33/3.58  3.98/4.04   3.52/3.87  5.03/4.25   4.05/4.19  5.95/4.76   10.6/7.0   b590 11.2/10.7
//   8-bit D = 129  3.37/4.33  4.00/4.86   3.57/4.59  5.05/5.25   4.16/5.03  6.09/6.18   11.0/10.1  b590 12.0/14.0
//   8-bit D = 101  4.25/4.23  5.68/4.86   4.59/4.55  7.19/5.19   5.76/5.04  9.01/6.02   17.2/9.7   b590 17.8/13.3
//   4-bit D = 202  4.97/3.46  6.76/3.86   5.42/3.68  8.29/4.17   7.00/4.07  10.8/4.7    20.9/7.2   b590 21.4/13.4
// Behind a pruning map a warp pools the rows that are left, half of them here, and the block walks over the gaps too:
//                  16 rows                30 rows                45 rows                64 rows
//   8-bit D = 128  2.97/3.39  3.15/4.08   3.23/4.27  4.33/4.46   4.24/4.46  5.56/4.68   4.66/4.50  7.03/4.94
//   4-bit D = 128  2.97/3.16  3.15/3.62   3.21/3.77  4.41/3.80   4.19/3.83  5.52/4.22   4.63/3.97  7.05/4.45
//   8-bit D = 256  3.11/3.45  3.44/4.31   3.49/4.32  4.73/4.48   4.61/4.56  6.12/4.94   5.17/4.71  7.86/5.23   b590 5.23/9.64  8.15/9.69
// Called and awaited, the host's part of 10 us hides half of such differences.
#pragma once

#include <cstdint>

namespace fbgemm_b200 {

struct FewBagsCall {
  int bits;          // of a column
  bool words;        // rows can be copied by four bytes (few_by_words)
  int units;         // copies that the widest tile of a row takes otherwise: halves or bytes
  int warp_chunks;   // chunks per lane of the kernel that would take the call (pick_variant)
  bool mapped;       // indices go through a pruning map
  int64_t tiles;     // of 128 columns
  int64_t bags;      // output rows
  int64_t beside;    // bags of launches on other streams
  int64_t rows;      // of all bags
};

inline bool few_bags_pay(const FewBagsCall& c, int64_t sms) {
  const auto average = [&](int64_t rows) { return c.rows / rows >= c.bags; };  // at least so many rows a bag
  const bool one_tile = c.tiles == 1;
  int64_t least, per_sm;  // rows a bag on average from which on blocks are faster, and up to how many of them an SM
  if (!c.words && c.warp_chunks >= 4) {  // warps whose rows in flight spill
    least = 16;
    per_sm = 4;
  } else if (!c.words && c.units > 64) {  // more than two copies a lane and row
    least = 60;
    per_sm = c.mapped ? 0 : 2;
  } else if (c.mapped) {
    least = c.words && c.bits == 2 ? 20 : c.words && c.bits == 8 ? 40 : 32;
    per_sm = average(!one_tile ? 40 : c.bits == 2 ? 28 : 56) ? 4 : 2;
  } else if (!c.words) {
    least = c.bits == 2 ? 16 : 20;
    per_sm = c.bits == 2 || average(30) ? 4 : 2;
  } else if (one_tile) {
    least = c.bits == 2 ? 1 : c.bits == 4 ? 20 : 32;
    per_sm = average(60) ? 8 : average(c.bits == 2 ? 20 : 32) ? 4 : 2;
  } else {
    least = 1;
    per_sm = average(c.bits == 2 ? 60 : 90) ? 8 : average(60) ? 6 : c.bits == 2 || average(20) ? 4 : 2;
  }
  return c.bags > 0 && average(least) && (c.bags + c.beside) * c.tiles <= per_sm * sms;
}

}  // namespace fbgemm_b200
