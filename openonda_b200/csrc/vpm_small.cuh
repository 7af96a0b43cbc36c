// vpm_small.cuh -- small all-pairs sums in one launch: pack, sweep and finalize together.
//
// A small sum is bound by latency, not by a pipe: with the tiled sweep, three launches in a
// row, a few blocks whose threads walk hundreds of sources each, and a finalize that sums the
// splits one after another.  Here a cluster of S blocks of four warps shares 32 R targets; each
// of its 4 S warps takes its own run of whole 32-source windows, reads those particles from
// the caller's arrays, rounds them into records in its own piece of shared memory (the next
// window's loads in flight under this one's sums) and sums them for all the targets.  The
// 4 S partial sums of a target are then added through distributed shared memory in a fixed
// order, and the same kernel writes the outputs.
//
// The pair terms, the FP32 windows (whole multiples of Op::kWindow sources from a window's
// start) and the FP64 carries are those of sweep_kernel, so results differ from it only by the
// order of FP64 additions.  No scratch memory.
//
// There is no order between clusters: one writes its targets' outputs while another still reads
// sources.  The outputs must therefore not overlap the inputs (the dispatch sends such calls
// through packed records instead).
#pragma once

#include <cooperative_groups.h>

#include "vpm_sweep.cuh"

namespace vpm {

constexpr int kSmallWarps = 4;
constexpr int kSmallThreads = 32 * kSmallWarps;
constexpr int kSmallWindow = 32;  // sources per staged window (one per lane)
constexpr int kSmallMaxCluster = 8;
static_assert(kSmallWindow == kCarryWindow, "a staged window is one carry window");

struct SmallArgs {
  const double* tpos;  // probe targets (m, 3), or the particles themselves
  const double* tstr;  // the targets' strengths and viscosities; null for probes
  const double* tnu;
  const double* pos;
  const double* str;
  const double* rad;
  int m, n;
  int windows_per_warp;
  int check_uniform;
  double *out, *out2;
};

__device__ __forceinline__ void set_record(double& e, double v) { e = v; }
__device__ __forceinline__ void set_record(float2& e, double v) {
  const float f = float(v);
  e = make_float2(f, f);
}

// One source particle as its lane holds it between the load and the store to shared memory.
struct SmallSrc {
  double x, y, z, s, ax, ay, az;
};

template <class Op, class V, int R, class Finalize>
__global__ void __launch_bounds__(kSmallThreads) small_sweep_kernel(const SmallArgs a) {
  namespace cg = cooperative_groups;
  using RecT = Rec<V>;
  constexpr int NV = Op::NV;
  constexpr int L = LaneTraits<V>::kLanes;
  constexpr int P = R / L;
  constexpr bool kCarry = (L == 2);
  constexpr int CW = Op::kWindow ? Op::kWindow : kCarryWindow;
  constexpr int TT = 32 * R;  // targets of the cluster
  static_assert(kSmallWindow % CW == 0, "carry windows tile a staged window");
  __shared__ __align__(128) RecT ring[kSmallWarps][kSmallWindow];
  __shared__ double part[kSmallWarps][NV][TT];
  __shared__ double total[NV][TT];

  cg::cluster_group cluster = cg::this_cluster();
  const int S = int(cluster.num_blocks()), rank = int(cluster.block_rank());
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int base = int(blockIdx.x / S) * TT;

  typename Op::TgtT tg[P];
  int64_t gi[R];
  V acc[P][NV];
  double car[kCarry ? R : 1][NV];
#pragma unroll
  for (int p = 0; p < P; ++p) {
    RecT rec[L];
    const RecT* recs[L];
#pragma unroll
    for (int k = 0; k < L; ++k) {
      const int r = p * L + k;
      const int t = base + r * 32 + lane;
      gi[r] = t;
      const int i = t < a.m ? t : a.m - 1;
      set_record(rec[k].x, a.tpos[3 * i]);
      set_record(rec[k].y, a.tpos[3 * i + 1]);
      set_record(rec[k].z, a.tpos[3 * i + 2]);
      // probes have no core and no strength, as their packed records
      set_record(rec[k].s, a.tstr ? a.rad[i] : 0.0);
      set_record(rec[k].ax, a.tstr ? a.tstr[3 * i] : 0.0);
      set_record(rec[k].ay, a.tstr ? a.tstr[3 * i + 1] : 0.0);
      set_record(rec[k].az, a.tstr ? a.tstr[3 * i + 2] : 0.0);
      set_record(rec[k].nu, 0.0);
      recs[k] = &rec[k];
    }
    tg[p] = Op::target(recs);
#pragma unroll
    for (int v = 0; v < NV; ++v) lane_zero(acc[p][v]);
  }
#pragma unroll
  for (int r = 0; r < (kCarry ? R : 1); ++r)
#pragma unroll
    for (int v = 0; v < NV; ++v) car[r][v] = 0.0;

  const int j0 = (rank * kSmallWarps + warp) * a.windows_per_warp * kSmallWindow;
  const int j1 = min(j0 + a.windows_per_warp * kSmallWindow, a.n);
  auto fetch = [&](int j) {
    SmallSrc q{};
    if (j < j1) {
      q.x = a.pos[3 * j];
      q.y = a.pos[3 * j + 1];
      q.z = a.pos[3 * j + 2];
      q.s = a.rad[j];
      q.ax = a.str[3 * j];
      q.ay = a.str[3 * j + 1];
      q.az = a.str[3 * j + 2];
      if (a.check_uniform && base == 0 && q.s != a.rad[0])
        atomicOr(&g_device_errors, VPM_DEVERR_NONUNIFORM_CORE);
    }
    return q;
  };
  SmallSrc next = fetch(j0 + lane);
  for (int j = j0; j < j1; j += kSmallWindow) {
    RecT rec;
    set_record(rec.x, next.x);
    set_record(rec.y, next.y);
    set_record(rec.z, next.z);
    set_record(rec.s, next.s);
    set_record(rec.ax, next.ax);
    set_record(rec.ay, next.ay);
    set_record(rec.az, next.az);
    set_record(rec.nu, 0.0);
    __syncwarp();  // the last window has been read
    ring[warp][lane] = rec;
    __syncwarp();
    next = fetch(j + kSmallWindow + lane);
    const int cnt = min(kSmallWindow, j1 - j);
    for (int w = 0; w < cnt; w += CW) {
      const int e = min(w + CW, cnt);
#pragma unroll 4
      for (int q = w; q < e; ++q) {
        const typename Op::SrcT src = Op::load(ring[warp][q]);
#pragma unroll
        for (int p = 0; p < P; ++p) Op::pair(tg[p], acc[p], src, &gi[p * L], j + q);
      }
      if constexpr (kCarry) {
#pragma unroll
        for (int p = 0; p < P; ++p)
#pragma unroll
          for (int v = 0; v < NV; ++v) {
#pragma unroll
            for (int k = 0; k < L; ++k) car[p * L + k][v] += lane_get(acc[p][v], k);
            lane_zero(acc[p][v]);
          }
      }
    }
  }

#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int v = 0; v < NV; ++v)
      part[warp][v][r * 32 + lane] = kCarry ? car[r][v] : lane_get(acc[r / L][v], r % L);
  cluster.sync();

  // this block's share of the targets: the 4 S partial sums in order, then the outputs
  const int share = (TT + S - 1) / S;
  const int t0 = rank * share;
  const int mine = min(share, TT - t0);
  for (int q = tid; q < NV * mine; q += kSmallThreads) {
    const int v = q / mine, t = t0 + q - v * mine;
    double sum = 0.0;
    for (int b = 0; b < S; ++b) {
      const double* remote = cluster.map_shared_rank(&part[0][v][t], b);
#pragma unroll
      for (int w = 0; w < kSmallWarps; ++w) sum += remote[w * NV * TT];
    }
    total[v][t - t0] = sum;
  }
  __syncthreads();
  if (tid < mine) {
    const int i = base + t0 + tid;
    if (i < a.m) {
      RecT rec;
      set_record(rec.ax, a.tstr ? a.tstr[3 * i] : 0.0);
      set_record(rec.ay, a.tstr ? a.tstr[3 * i + 1] : 0.0);
      set_record(rec.az, a.tstr ? a.tstr[3 * i + 2] : 0.0);
      set_record(rec.nu, a.tnu ? a.tnu[i] : 0.0);
      double v[NV];
#pragma unroll
      for (int k = 0; k < NV; ++k) v[k] = total[k][tid];
      Finalize::write(v, &rec, a.out + 3 * int64_t(i), a.out2 ? a.out2 + 3 * int64_t(i) : nullptr);
    }
  }
  cluster.sync();  // no block leaves while its partial sums are read
}

}  // namespace vpm
