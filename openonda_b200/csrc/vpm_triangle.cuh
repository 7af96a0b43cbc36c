// vpm_triangle.cuh -- FP32-compensated both-sides sums in one launch of equal blocks.
//
// The tile pairs, their orientation (the lower tile holds the targets), the batches and the FP32
// windows are rot_sweep_kernel's (vpm_rot.cuh), so every FP32 sum has the same terms in the same
// order; only FP64 additions are ordered differently.  The schedule is the one of
// vpm_circle.cuh: that kernel launches diagonals one after another, each launch ending in a
// partly filled wave, while here the tile pairs (I, J), J > I, of all I one after another are cut
// into shares (vpm_shares.cuh), one block each.  The unit is two batches (64 sources), the span of
// the longest target window, so that windows start where they do in a tile pair of its own.
//
// Source sums of tile I's list go to a set of their own for the particles after tile I, a block's
// target sums to the set of its place among the blocks that share the list: every element is
// written once, none is zeroed.  The diagonal tiles are rot_sweep_kernel<Op, true>'s.
//
// Memory: about nt / 2 sets of NV values per particle (at n = 65536 and T = 768, 240 MB for the
// fused sum), written and read once.
//
// Bound: the FP32 pipe, as rot_sweep_kernel.  Measured against the launches of its first form (Gpairs/s at 32768 /
// 65536 / 131072 particles): velocity 1531 / 1685 / 1860 -> 1750 / 1821 / 1858, PSE 1882 / 2078 /
// 2322 -> 2167 / 2272 / 2331, fused 827 / 935 / 962 -> 892 / 972 / 989, LES 583 / 616 / 627 -> 611
// / 634 / 642, adjoint 393 / 413 / 421 -> 409 / 423 / 421, with PSE 272 / 278 / 279 -> 279 / 283 /
// 280.  FP64 (vpm_circle.cuh), fused / velocity / PSE / LES at 50000: 408 / 663 / 831 / 224 -> 458
// / 759 / 955 / 260.
#pragma once

#include "vpm_rot.cuh"
#include "vpm_shares.cuh"

namespace vpm {

constexpr int kTriUnit = 64;  // sources

struct TriArgs {
  const void* rec;
  int n;
  int nt;
  Shares shares;   // in units
  double* target;  // [sets][NV][n]
  double* source;  // tile I's set: [NV][n - (I + 1) T]
};

template <class Op>
__global__ void __launch_bounds__(kRotThreads, Op::kMinBlocks)
rot_triangle_kernel(const TriArgs a) {
  using Record = typename Op::Record;
  using Lane = typename Op::Lane;
  constexpr int NV = Op::NV;
  constexpr int P = Op::kP;
  constexpr int T = rot_tile<Op>();
  constexpr int NJ = Op::kSymFrom;
  static_assert(T % kTriUnit == 0, "tiles are whole units");
  static_assert(kTriUnit % (Op::kTgtWindowLong > 0 ? Op::kTgtWindowLong : 1) == 0,
                "units are whole target windows");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  double* car = reinterpret_cast<double*>(smem_raw);  // [NV][T]
  float2* jbuf = reinterpret_cast<float2*>(smem_raw + size_t(T) * NV * sizeof(double));
  const Record* rec = static_cast<const Record*>(a.rec);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const TriLists lists(a.n, T, kTriUnit);
  int64_t w = a.shares.begin(blockIdx.x);
  const int64_t wend = a.shares.end(blockIdx.x);
  int buf = 0;
  int lt[2 * P];
  rot_rows<P>(lt, warp, lane);

  while (w < wend) {
    const int I = lists.tile(w);
    const int64_t first = lists.start(I);
    const int u0 = int(w - first);
    const int u1 = u0 + int(min(int64_t(lists.length(I) - u0), wend - w));
    w += u1 - u0;
    const int i0 = I * T;

    // each thread zeroes, folds into and writes out its own rows of the carries
    typename Op::TgtT tg[P];
    float2 acc[P][NV];
#pragma unroll
    for (int p = 0; p < P; ++p) {
      const Record* recs[2] = {rec + i0 + lt[2 * p], rec + i0 + lt[2 * p + 1]};
      tg[p] = Op::target(recs);
      if constexpr (Op::kUniformCore) Op::uniform_core(tg[p], rec);
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        acc[p][v] = make_float2(0.f, 0.f);
        car[v * T + lt[2 * p]] = 0.0;
        car[v * T + lt[2 * p + 1]] = 0.0;
      }
    }
    // tile I's source set, at the first particle after the tile
    double* out = a.source + int64_t(NV) * lists.before(I, a.n, T);
    const int len = a.n - i0 - T;

    const int b0 = 2 * u0, b1 = 2 * u1;  // batches, T / 32 in a tile
    auto place = [&](int b, int& b_in_tile) {
      const int t = b / (T / 32);
      b_in_tile = b - t * (T / 32);
      return (I + 1 + t) * T + b_in_tile * 32;
    };
    int bt;
    int j = place(b0, bt);
    Lane nxt = Op::load_lane(rec, j + lane, a.n);
    for (int b = b0; b < b1; ++b) {
      const Lane cur = nxt;
      const int jb0 = j, bin = bt;
      const int have = min(32, a.n - jb0);
      if (b + 1 < b1) {
        j = place(b + 1, bt);
        nxt = Op::load_lane(rec, j + lane, a.n);
      }
      if (have > 0) {
        float2* jb = jbuf + buf * (NJ * kRotWarps * 32);
        if constexpr (Op::kJBufs == 2) buf ^= 1;
        rot_batch<Op, false>(cur, tg, acc, lt, car, jb, i0, jb0, bin, warp, lane);
        __syncthreads();  // the batch's source-side sums are complete
        rot_combine<Op>(jb, have, tid, [&](int v, int jj, double sum) {
          out[int64_t(v) * len + (jb0 - i0 - T) + jj] = -sum;
        });
        if constexpr (Op::kJBufs == 1) __syncthreads();
      }
    }
    // the last tile may end in half a long window
    if constexpr (Op::kTgtWindowLong > 0)
      rot_fold<Op, false>(car, acc, lt, [](int v) { return Op::long_fold(v); });

    double* sum = a.target + int64_t(int(blockIdx.x) - a.shares.block_of(first)) * NV * a.n;
#pragma unroll
    for (int q = 0; q < 2 * P; ++q)
#pragma unroll
      for (int v = 0; v < NV; ++v) sum[int64_t(v) * a.n + i0 + lt[q]] = car[v * T + lt[q]];
  }
}

}  // namespace vpm
