// vpm_circle.cuh -- FP64 self sums with each unordered pair once, in one launch of equal blocks.
//
// The pair terms and the travel of a source around the warp are those of rot64_sweep_kernel
// (vpm_rot.cuh); what differs is the schedule.  That kernel gives a block one pair of tiles,
// keeps one writer per accumulator element by launching the diagonals one after another, and
// adds into accumulators: below about 24576 particles its launches leave most of the GPU idle.
// Here
//
//   * particles form nt tiles of T = 128 R, and target tile I meets the source tiles I, I + 1,
//     .., I + nt / 2 (mod nt): a circle, so all target tiles have the same list of sources (for
//     even nt its last tile is met by the tiles I < nt / 2 only).  The tile's own sources are
//     visited one-sided;
//   * all lists, in batches of 32 sources and one after another, are cut into shares
//     (vpm_shares.cuh), one block each.  A block walks its share, which may end one list and
//     begin the next;
//   * nothing is accumulated in memory: for target tile I, source j's sums go to the set of the
//     distance of their tiles, and a block's target sums to the set of its place among the
//     blocks that share the list.  Every element that is read has been written exactly once (the
//     finalize passes by the values without source sums), so no set is zeroed, and the finalize
//     adds the sets in a fixed order.
//
// A target past n (in the last tile) is a particle far away without strength, as a source past n
// is: the pair's terms underflow to zero on both sides.
//
// Memory: nt / 2 sets of source sums, and as many sets of target sums as blocks share one list (the
// small shares of the last lists: up to 128 below about 16384 particles, though most tiles write
// a few of them).  The fused sum asks for 81 MB at 8192 particles (136 sets), 171 MB at 16384 (144);
// the adjoint for 3970 MB at 131072.  Written and read once: about 1 % of the sweep.  Past 4 GB
// (stretching from about 297000 particles, adjoint 137000, with PSE 120000) the sums take several
// launches (vpm_rot.cuh).
//
// Bound: the FP64 pipe at 8 warps per SM (58 operations per unordered pair of the fused sum, root
// included).  Measured against the one-sided sweeps (us, velocity / fused / stretching / PSE /
// LES / adjoint / with PSE): 153 / 234 / 220 / 138 / 440 / 550 / 699 -> 109 / 182 / 139 / 91 / 282
// / 389 / 570 at 8192 particles, 549 / 780 / 744 / 515 / 1555 / 2032 / 2599 -> 375 / 627 / 476 /
// 305 / 1060 / 1425 / 2114 at 16384; stretching and adjoint at 131072 44.6 / 122.7 -> 28.8 / 86.2
// ms (with PSE, in several launches there, 157.7 -> 125.9).
#pragma once

#include "vpm_rot.cuh"
#include "vpm_shares.cuh"

namespace vpm {

struct Sweep64Args {
  const void* rec;
  int n;
  Shares shares;   // in batches
  double* target;  // [sets][NV][n]
  double* source;  // the source sums, where the lists say
};

// The lists: target tile I's has (1 + distances) tiles of `per` batches, its own tile first.
struct CircleLists {
  static constexpr bool kOwnTile = true;
  int nt, half, per;
  __host__ __device__ CircleLists(int64_t n, int tile) {
    nt = int((n + tile - 1) / tile);
    half = nt / 2;
    per = tile / 32;
  }
  // the t-th tile of tile I's list
  __device__ __forceinline__ int source_tile(int I, int t) const {
    const int J = I + t;
    return J < nt ? J : J - nt;
  }
  // source sums of particle j, met by tile I as the t-th of its list: set t - 1, [NV][n]
  __device__ __forceinline__ double* source_sums(double* source, int nv, int, int t, int j,
                                                 int64_t n, int, int64_t& stride) const {
    stride = n;
    return source + int64_t(t - 1) * nv * n + j;
  }
  // tiles with the full half circle; the others (even nt) stop one short
  __host__ __device__ int full() const { return (nt % 2 == 0) ? half : nt; }
  __host__ __device__ int length(int I) const { return (1 + half - (I < full() ? 0 : 1)) * per; }
  __host__ __device__ int64_t start(int I) const {
    const int f = I < full() ? I : full();
    return (int64_t(f) * (1 + half) + int64_t(I - f) * half) * per;
  }
  __host__ __device__ int64_t total() const { return start(nt); }
  // the tile whose list holds batch w
  __host__ __device__ int tile(int64_t w) const {
    const int64_t first = start(full());
    if (w < first) return int(w / (int64_t(1 + half) * per));
    return full() + int((w - first) / (int64_t(half) * per));
  }
};

// The triangle of vpm_shares.cuh in the same form (batches of 32): every tile pair with the lower
// tile as target, the diagonal tiles left to rot64_sweep_kernel<Op, true>.
struct TriLists64 : TriLists {
  static constexpr bool kOwnTile = false;
  __host__ __device__ TriLists64(int64_t n, int tile) : TriLists(n, tile, 32) {}
  __device__ __forceinline__ int source_tile(int I, int t) const { return I + 1 + t; }
  __device__ __forceinline__ double* source_sums(double* source, int nv, int I, int, int j,
                                                 int64_t n, int tile, int64_t& stride) const {
    stride = n - int64_t(I + 1) * tile;
    return source + int64_t(nv) * before(I, n, tile) + j - int64_t(I + 1) * tile;
  }
};

template <class Op>
constexpr size_t lists64_smem_bytes() {
  return size_t(2 * Op::kSymFrom + Op::NV * 2 * Op::kP) * kRotThreads * sizeof(double);
}

template <class Op, class Lists>
__global__ void __launch_bounds__(kRotThreads, Op::kMinBlocks)
rot64_lists_kernel(const Sweep64Args a) {
  using Record = typename Op::Record;
  constexpr int NV = Op::NV;
  constexpr int NJ = Op::kSymFrom;  // values with a source side: the first NJ
  constexpr int R = 2 * Op::kP;
  constexpr int T = rot_tile<Op>();
  constexpr int WT = kRotWarps * 32;
  constexpr int PER = T / 32;
  static_assert(T == R * WT, "a tile is the block's lanes times their targets");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  double* jbuf = reinterpret_cast<double*>(smem_raw);  // [2][NJ][WT]
  // the thread's sums over the source tiles it is done with, [NV][R][WT]: a sum in registers runs
  // over one tile only, so that its rounding grows no further than in a tile pair of its own
  double* car = jbuf + 2 * NJ * WT + threadIdx.x;
  const Record* rec = static_cast<const Record*>(a.rec);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int src_lane = (lane + 1) & 31;
  const Lists lists(a.n, T);
  int64_t w = a.shares.begin(blockIdx.x);
  const int64_t wend = a.shares.end(blockIdx.x);
  int buf = 0;

  while (w < wend) {
    const int I = lists.tile(w);
    const int64_t first = lists.start(I);
    const int b0 = int(w - first);
    const int left = int(wend - w);
    const int b1 = min(lists.length(I), b0 + left);
    w += b1 - b0;

    typename Op::TgtT tg[R];
    int64_t ti[R];
    double acc[R][NV];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      ti[r] = int64_t(I) * T + warp * 32 * R + r * 32 + lane;
      tg[r] = Op::target(rec, ti[r], a.n);
      if constexpr (Op::kUniformCore) Op::uniform_core(tg[r], rec);
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        acc[r][v] = 0.0;
        car[(v * R + r) * WT] = 0.0;
      }
    }
    auto fold = [&] {
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          car[(v * R + r) * WT] += acc[r][v];
          acc[r][v] = 0.0;
        }
    };

    // first source of batch b of this list, and how many it holds
    auto place = [&](int b, int& j0) {
      j0 = lists.source_tile(I, b / PER) * T + (b % PER) * 32;
      return min(32, max(0, a.n - j0));
    };
    int j0;
    int cnt = place(b0, j0);
    typename Op::SrcT nxt;
    if (Op::kPrefetch) nxt = Op::load(rec, j0 + lane, j0 + cnt);
    for (int b = b0; b < b1; ++b) {
      const int j = j0, have = cnt;
      typename Op::SrcT cur = Op::kPrefetch ? nxt : Op::load(rec, j + lane, j + have);
      if (b + 1 < b1) {
        cnt = place(b + 1, j0);
        if (Op::kPrefetch) nxt = Op::load(rec, j0 + lane, j0 + cnt);
      }
      if (Lists::kOwnTile && b < PER) {  // the tile's own sources, one-sided
#pragma unroll 1
        for (int st = 0; st < 32; ++st) {
#pragma unroll
          for (int r = 0; r < R; ++r)
            Op::diag(tg[r], acc[r], cur, &ti[r], j + ((lane + st) & 31));
          Op::shuffle(cur, src_lane);
        }
        if constexpr (NJ < NV) {
          // a symmetric sum taken once per unordered pair elsewhere: the own tile visits every
          // ordered pair, so it counts half (the finalize doubles the sum)
          if (b == PER - 1 || b == b1 - 1) {
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
              for (int v = NJ; v < NV; ++v) acc[r][v] *= 0.5;
          }
        }
        continue;
      }
      if (b % PER == 0) fold();  // the next tile
      if (have == 0) continue;  // the ragged end of the last tile (the whole block)
      double jv[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) jv[v] = 0.0;
#pragma unroll Op::kUnroll
      for (int st = 0; st < 32; ++st) {
        Op::pairs(tg, acc, jv, cur);
        Op::shuffle(cur, src_lane);
#pragma unroll
        for (int v = 0; v < NJ; ++v)
          if (Op::carried(v)) jv[v] = __shfl_sync(0xffffffffu, jv[v], src_lane);
      }
      // the warps' sums of the batch's sources, added over the warps in a fixed order; with two
      // buffers one barrier a batch is enough (a buffer is written again two batches later)
      double* jb = jbuf + buf * (NJ * WT);
      buf ^= 1;
#pragma unroll
      for (int v = 0; v < NJ; ++v) jb[v * WT + warp * 32 + lane] = jv[v];
      __syncthreads();
      int64_t stride;
      double* out = lists.source_sums(a.source, NV, I, b / PER, j, a.n, T, stride);
      for (int q = tid; q < 32 * NJ; q += kRotThreads) {
        const int v = q >> 5, jj = q & 31;
        if (!Op::carried(v)) continue;
        double sum = 0.0;
#pragma unroll
        for (int k = 0; k < kRotWarps; ++k) sum += jb[v * WT + k * 32 + jj];
        if (jj < have) out[int64_t(v) * stride + jj] = -sum;
      }
    }

    double* out = a.target + int64_t(int(blockIdx.x) - a.shares.block_of(first)) * NV * a.n;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (ti[r] < a.n) {
#pragma unroll
        for (int v = 0; v < NV; ++v)
          out[int64_t(v) * a.n + ti[r]] = car[(v * R + r) * WT] + acc[r][v];
      }
    }
  }
}

// The sets that hold particle i's sums (finalize_sets_kernel): of target sums the blocks that
// share its tile's list, of source sums the distances at which another tile meets it.
struct CircleSets {
  CircleLists lists;
  Shares shares;
  int tile, tsets;
  __device__ __forceinline__ void ranges(int64_t i, int& t, int& s) const {
    const int I = int(i / tile);
    t = shares.sharing(lists.start(I), lists.length(I));
    // source sums: tile I - k has I in its list; for even nt, k = nt / 2 only from I >= nt / 2
    s = lists.half - ((lists.nt % 2 == 0 && I < lists.half) ? 1 : 0);
  }
  int64_t n;
  template <int NV>
  __device__ __forceinline__ const double* source_set(const double* acc, int q, int64_t i,
                                                      int64_t&) const {
    return acc + int64_t(tsets + q) * NV * n + i;
  }
};

}  // namespace vpm
