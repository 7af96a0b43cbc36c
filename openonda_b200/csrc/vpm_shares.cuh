// vpm_shares.cuh -- cutting one long list of work into blocks' shares.
//
// The one-launch schedule (vpm_circle.cuh) lays all lists end to end and cuts
// the line into shares.  One equal share per resident block leaves the end to the slowest: blocks
// of the same work differ by some percent (their place on the chip, what runs beside them), and
// the sweep waits for the last.  So as many blocks as are resident get a large share first, and
// what is left is cut into small ones that the hardware hands out as blocks finish.
#pragma once

#include <cstdint>

namespace vpm {

struct Shares {
  int64_t total;  // units of work
  int64_t cut;    // large * count: where the small shares begin
  int large, small, count;

  // total units on `slots` resident blocks: 85 % of a block's part at once, the rest in about three
  // pieces per resident block.  Measured (stretching / adjoint at 131072, Gpairs/s): one equal
  // share per block 588 / 191, eight 607 / 199, 85 % and three pieces 597 / 199; at 32768 575 / 188,
  // 590 / 196, 579 / 195; many pieces add sets of target sums at small n.
  static Shares make(int64_t total, int64_t slots) {
    Shares s{total, 0, 0, 1, 0};
    const int64_t large = total * 85 / 100 / slots;
    if (large > 0) {
      s.large = int(large);
      s.count = int(slots);
      s.cut = large * slots;
    }
    const int64_t left = total - s.cut;
    const int64_t pieces = slots * 3;
    s.small = int((left + pieces - 1) / pieces);
    if (s.small < 1) s.small = 1;
    return s;
  }
  __host__ __device__ int blocks() const { return count + int((total - cut + small - 1) / small); }
  __host__ __device__ int64_t begin(int block) const {
    return block < count ? int64_t(block) * large : cut + int64_t(block - count) * small;
  }
  __host__ __device__ int64_t end(int block) const {
    const int64_t e = begin(block) + (block < count ? large : small);
    return e < total ? e : total;
  }
  __host__ __device__ int block_of(int64_t w) const {
    return w < cut ? int(w / large) : count + int((w - cut) / small);
  }
  // blocks that share the units [first, first + length)
  __host__ __device__ int sharing(int64_t first, int length) const {
    return length > 0 ? block_of(first + length - 1) - block_of(first) + 1 : 0;
  }
};

// Most blocks that share one list: the sets of target sums.
template <class Lists>
int target_sets(const Lists& lists, const Shares& shares) {
  int most = 1;
  for (int I = 0; I < lists.nt; ++I) {
    const int k = shares.sharing(lists.start(I), lists.length(I));
    if (k > most) most = k;
  }
  return most;
}

}  // namespace vpm
