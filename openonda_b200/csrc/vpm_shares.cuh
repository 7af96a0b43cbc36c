// vpm_shares.cuh -- cutting one long list of work into blocks' shares.
//
// The one-launch schedules (vpm_circle.cuh, vpm_triangle.cuh) lay all lists end to end and cut
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
  // pieces per resident block.  Measured (FP32c fused / velocity / LES sums at 131072, Gpairs/s):
  // one equal share per block 941 / 1800 / 598, eight 981 / 1849 / 630, 75 % and four pieces 988 /
  // 1856 / 641, 85 % and three 989 / 1858 / 642, 85 % and six 992 / 1857 / 630; many pieces add
  // sets of target sums at small n (velocity at 32768: 1750 with this rule, 1469 with 32 shares).
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

// The lists of a triangle of tile pairs: tile I's holds the tiles I + 1 .. nt - 1, `per` units of
// sources each and `last` in the last.
struct TriLists {
  int nt, per, last;
  __host__ __device__ TriLists(int64_t n, int tile, int unit) {
    nt = int((n + tile - 1) / tile);
    per = tile / unit;
    last = int((n - int64_t(nt - 1) * tile + unit - 1) / unit);
  }
  __host__ __device__ int64_t start(int I) const {
    return int64_t(I) * last + int64_t(per) * (int64_t(I) * (nt - 2) - int64_t(I) * (I - 1) / 2);
  }
  __host__ __device__ int length(int I) const {
    return I < nt - 1 ? (nt - 2 - I) * per + last : 0;
  }
  __host__ __device__ int64_t total() const { return start(nt - 1); }
  // the tile whose list holds unit w
  __host__ __device__ int tile(int64_t w) const {
    int lo = 0, hi = nt - 2;
    while (lo < hi) {
      const int mid = (lo + hi + 1) / 2;
      if (start(mid) <= w)
        lo = mid;
      else
        hi = mid - 1;
    }
    return lo;
  }
  // particles of the source sets before tile I's
  __host__ __device__ int64_t before(int I, int64_t n, int tile) const {
    return int64_t(I) * n - int64_t(tile) * (int64_t(I) * (I + 1) / 2);
  }
};

// The sets that hold particle i's sums (finalize_sets_kernel): the blocks that share its tile's
// list, the parts of the diagonal tiles, and the lists of the tiles before its own.
struct TriSets {
  TriLists lists;
  Shares shares;
  int tile, diagonal;  // diagonal: sets [0, diagonal) are the diagonal tiles'
  int64_t n;
  const double* source;
  __device__ __forceinline__ void ranges(int64_t i, int& t, int& s) const {
    const int I = int(i / tile);
    t = diagonal + shares.sharing(lists.start(I), lists.length(I));
    s = I;
  }
  template <int NV>
  __device__ __forceinline__ const double* source_set(const double*, int q, int64_t i,
                                                      int64_t& stride) const {
    stride = n - int64_t(q + 1) * tile;
    return source + NV * lists.before(q, n, tile) + i - int64_t(q + 1) * tile;
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
