// Copies between a caller's pageable memory and page-locked staging blocks by
// several host threads.
//
// One thread copies at about 17 GB/s, a third of what the link moves: the 5.1 MB
// of rows of a 10 000-bag call took 300 us to leave the staging block after a
// transfer of 93 us.  A few helpers bring the copy down to the transfer's time,
// and the transfers of a call's parts overlap the copies of the others.
#pragma once

#include <cstddef>
#include <functional>

namespace fbgemm_b200 {

struct CopySlice {
  void* dst;
  const void* src;
  size_t bytes;
  int part;  // 0, 1, ... < kCopyParts, not decreasing from slice to slice
};
constexpr int kCopyParts = 16;

// Copies all slices.  Before the slices of part p are copied ready(p) is called, and once they are copied done(p), both
// on the calling thread, part after part (a part may have no slices); they return false to end the whole copy early.
// With `ahead` the slices of all parts may be copied at once (ready() is not called), otherwise only those of parts
// that are ready.  Returns false if a callback did.
bool copy_slices(const CopySlice* slices, int count, int parts, bool ahead, const std::function<bool(int)>& ready,
                 const std::function<bool(int)>& done);

}  // namespace fbgemm_b200
