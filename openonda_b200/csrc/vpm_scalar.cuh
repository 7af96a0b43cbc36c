// vpm_scalar.cuh -- FP64 scalar diagnostics (kinetic energy, enstrophy, helicity) with each
// unordered pair evaluated once.
//
// The pair terms of the three sums are symmetric under i <-> j, and only the sum over all
// pairs is wanted, so a pair is visited once and adds one scalar: no per-target vectors and no
// source-side sums (the one-sided sweeps visit it twice and carry three sums per target).
//
// Schedule: particles form nt tiles of T = 128 R.  Target tile I meets the source tiles I,
// I + 1, .., I + nt/2 (mod nt): a circle, so every target tile has the same work (for even nt
// the last one, I + nt/2, is taken by the tiles I < nt/2 only).  Its list of sources, in pieces
// of kScalarPiece records, is cut into `splits` equal parts, one block each.  The tile's own
// records (piece index below T / kScalarPiece) are visited in both orders and count half.  A
// block keeps R targets per thread in registers, stages the pieces in a two-stage ring of bulk
// copies as sweep_kernel does, and leaves one partial sum; scalar_total_kernel adds the partials
// in a fixed order.  From the threads' sums on, every addition carries its rounding error along
// (two-sum), so the total is rounded once or twice instead of some twenty times.
//
// Bound: the FP64 pipe (28 / 21 / 28 operations per unordered pair).  Measured against the
// one-sided sweeps (us, kinetic energy / enstrophy / helicity): 2311 / 1819 / 2173 -> 1069 / 779
// / 1022 at 32768 particles, 69 / 59 / 67 -> 25 / 20 / 25 at 4096.  Two targets per thread and
// eight sources unrolled; four sources 1078 / 815 / 1046, two 1100 / 877 / 1070, one 1147 / 941 /
// 1099, four targets 1139 / 877 / 1109 at 32768.
#pragma once

#include "vpm_sweep.cuh"

namespace vpm {

constexpr int kScalarThreads = 128;
constexpr int kScalarPiece = 64;  // source records per staged piece

// Each operator adds one pair's symmetric term to acc; SELF: i == j adds what the reference's
// own double loop adds there.
struct ScalarKe {  // (1/16 pi) sum_{i != j} of the term (OpKe)
  template <bool SELF>
  __device__ __forceinline__ static void pair(const Tgt<double>& t, double& acc,
                                              const Src<double>& s, bool same) {
    const double rx = t.x - s.x, ry = t.y - s.y, rz = t.z - s.z;
    double sg, s2;
    pair_core<false>(t, s, sg, s2);
    const double x = fma(rx, rx, fma(ry, ry, fma(rz, rz, s2)));
    const double y = rsqrt_lane<false>(x);
    const double y3 = (y * y) * y;
    const double w = fma(s2, y3, y);
    const double p1 = fma(t.ax, s.ax, fma(t.ay, s.ay, t.az * s.az));
    const double ri = fma(rx, t.ax, fma(ry, t.ay, rz * t.az));
    const double rj = fma(rx, s.ax, fma(ry, s.ay, rz * s.az));
    const double next = fma(y3, ri * rj, fma(w, p1, acc));
    acc = (SELF && same) ? acc : next;
  }
};

struct ScalarEns {  // all pairs, i == j among them (OpEns)
  template <bool SELF>
  __device__ __forceinline__ static void pair(const Tgt<double>& t, double& acc,
                                              const Src<double>& s, bool) {
    const double rx = t.x - s.x, ry = t.y - s.y, rz = t.z - s.z;
    double sg, s2;
    pair_core<false>(t, s, sg, s2);
    const double x = fma(rx, rx, fma(ry, ry, fma(rz, rz, s2)));
    const double y = rsqrt_lane<false>(x);
    const double k = fma(2.2, s2, x) * ((y * y) * y);
    acc = fma(k, fma(t.ax, s.ax, fma(t.ay, s.ay, t.az * s.az)), acc);
  }
};

struct ScalarHel {  // a_i . sum_j g (r x a_j) (OpVel dotted with the target's strength)
  template <bool SELF>
  __device__ __forceinline__ static void pair(const Tgt<double>& t, double& acc,
                                              const Src<double>& s, bool) {
    const double rx = t.x - s.x, ry = t.y - s.y, rz = t.z - s.z;
    double sg, s2;
    pair_core<false>(t, s, sg, s2);
    const double x = fma(rx, rx, fma(ry, ry, fma(rz, rz, s2)));
    const double y = rsqrt_lane<false>(x);
    const double y2 = y * y;
    const double g = fma(1.5, s2, x) * ((y2 * y2) * y);
    const double cx = fma(ry, s.az, -(rz * s.ay));  // r x a_j
    const double cy = fma(rz, s.ax, -(rx * s.az));
    const double cz = fma(rx, s.ay, -(ry * s.ax));
    acc = fma(g, fma(t.ax, cx, fma(t.ay, cy, t.az * cz)), acc);
  }
};

// A sum and the error of its rounding so far.
struct TwoSum {
  double hi, lo;
  __device__ __forceinline__ void add(double x, double low) {
    const double s = __dadd_rn(hi, x);
    const double b = __dadd_rn(s, -hi);
    lo = __dadd_rn(lo, __dadd_rn(low, __dadd_rn(__dadd_rn(hi, -__dadd_rn(s, -b)),
                                                __dadd_rn(x, -b))));
    hi = s;
  }
};

// The warp's sums in lane 0, in a fixed order.
__device__ __forceinline__ void warp_total(TwoSum& t) {
#pragma unroll
  for (int w = 16; w > 0; w >>= 1) {
    const double hi = __shfl_down_sync(0xffffffffu, t.hi, w);
    const double lo = __shfl_down_sync(0xffffffffu, t.lo, w);
    t.add(hi, lo);
  }
}

struct ScalarArgs {
  const Rec<double>* rec;
  int64_t n;
  int nt;      // target tiles
  int chunk;   // source pieces per block
  double* partial;  // [gridDim.y][gridDim.x][2]: the blocks' sums and their rounding errors
};

template <class Op, int R>
__global__ void __launch_bounds__(kScalarThreads, R == 1 ? 6 : 4)
scalar_pairs_kernel(const ScalarArgs a) {
  constexpr int T = kScalarThreads * R;
  constexpr int S = T / kScalarPiece;  // pieces per tile
  constexpr int STAGES = 2;
  constexpr uint32_t kRecBytes = sizeof(Rec<double>);
  __shared__ __align__(128) Rec<double> ring[STAGES][kScalarPiece];
  __shared__ __align__(8) uint64_t full_bar[STAGES];
  __shared__ TwoSum red[kScalarThreads / 32];

  const int tid = threadIdx.x;
  const int I = blockIdx.x;
  const int half = a.nt / 2;
  // this tile's pieces: its own tile and the half circle after it
  const int tiles = 1 + half - ((a.nt % 2 == 0 && I >= half && half > 0) ? 1 : 0);
  const int p0 = blockIdx.y * a.chunk;
  const int p1 = min(p0 + a.chunk, tiles * S);

  Tgt<double> tg[R];
  int64_t ti[R];
  double acc[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    ti[r] = int64_t(I) * T + r * kScalarThreads + tid;
    const Rec<double>* rp = a.rec + (ti[r] < a.n ? ti[r] : a.n - 1);
    tg[r] = make_tgt(&rp);
    acc[r] = 0.0;
  }
  if (tid == 0) {
#pragma unroll
    for (int s = 0; s < STAGES; ++s) mbar_init(&full_bar[s], 1);
    fence_mbar_init();
  }
  __syncthreads();

  // first record of piece p and how many it holds (none in the ragged tail of the last tile)
  auto place = [&](int p, int64_t& j0) {
    int J = I + p / S;
    if (J >= a.nt) J -= a.nt;
    j0 = int64_t(J) * T + int64_t(p % S) * kScalarPiece;
    const int64_t left = a.n - j0;
    return int(left < kScalarPiece ? (left > 0 ? left : 0) : kScalarPiece);
  };
  auto issue = [&](int p) {
    int64_t j0;
    const int cnt = place(p, j0);
    const int s = (p - p0) % STAGES;
    mbar_arrive_expect_tx(&full_bar[s], uint32_t(cnt) * kRecBytes);
    if (cnt > 0) bulk_load_g2s(ring[s], a.rec + j0, uint32_t(cnt) * kRecBytes, &full_bar[s]);
  };
  if (tid == 0) {
    for (int p = p0; p < p0 + STAGES && p < p1; ++p) issue(p);
  }

  int failed_at = -1;
  for (int p = p0; p < p1; ++p) {
    const int s = (p - p0) % STAGES;
    const bool ok = mbar_wait_bounded(&full_bar[s], uint32_t(((p - p0) / STAGES) & 1));
    int64_t j0;
    const int cnt = place(p, j0);
    if (ok) {
      if (p < S) {
        for (int j = 0; j < cnt; ++j) {
          const Src<double> src = load_src<double>(ring[s][j]);
#pragma unroll
          for (int r = 0; r < R; ++r)
            Op::template pair<true>(tg[r], acc[r], src, ti[r] == j0 + j);
        }
        if (p == min(S, p1) - 1) {  // the last of the tile's own pieces here: both orders seen
#pragma unroll
          for (int r = 0; r < R; ++r) acc[r] *= 0.5;
        }
      } else {
#pragma unroll 8
        for (int j = 0; j < cnt; ++j) {
          const Src<double> src = load_src<double>(ring[s][j]);
#pragma unroll
          for (int r = 0; r < R; ++r) Op::template pair<false>(tg[r], acc[r], src, false);
        }
      }
    }
    if (__syncthreads_or(!ok)) {
      failed_at = p;
      break;
    }
    if (tid == 0 && p + STAGES < p1) issue(p + STAGES);
  }
  if (failed_at >= 0) {
    // let the copies this block still has in flight land before the block exits
    if (tid == 0) {
      const int last = (failed_at + STAGES < p1) ? failed_at + STAGES : p1;
      for (int p = failed_at; p < last; ++p)
        mbar_wait_bounded(&full_bar[(p - p0) % STAGES], uint32_t(((p - p0) / STAGES) & 1));
    }
    return;
  }

  TwoSum sum{0.0, 0.0};
#pragma unroll
  for (int r = 0; r < R; ++r) sum.add(ti[r] < a.n ? acc[r] : 0.0, 0.0);
  warp_total(sum);
  if ((tid & 31) == 0) red[tid >> 5] = sum;
  __syncthreads();
  if (tid == 0) {
#pragma unroll
    for (int w = 1; w < kScalarThreads / 32; ++w) sum.add(red[w].hi, red[w].lo);
    double* out = a.partial + 2 * (int64_t(blockIdx.y) * gridDim.x + I);
    out[0] = sum.hi;
    out[1] = sum.lo;
  }
}

// out = scale * sum of the blocks' partials, in a fixed order.
__global__ void __launch_bounds__(1024)
scalar_total_kernel(const double* __restrict__ partial, int count, double scale,
                    double* __restrict__ out) {
  __shared__ TwoSum red[32];
  TwoSum sum{0.0, 0.0};
  for (int i = threadIdx.x; i < count; i += 1024) sum.add(partial[2 * i], partial[2 * i + 1]);
  warp_total(sum);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x < 32) {
    sum = red[threadIdx.x];
    warp_total(sum);
    if (threadIdx.x == 0) {
      // (hi + lo) scale, rounded once; a sum that is not finite has no rounding error
      const double p = __dmul_rn(sum.hi, scale);
      const double e = fma(sum.hi, scale, -p) + sum.lo * scale;
      out[0] = isfinite(p) ? p + e : p;
    }
  }
}

}  // namespace vpm
