// vpm_sets.cuh -- finalize pass over many sets of partial sums.
//
// acc[set][value][n]: a block takes 32 particles, its kSetLanes warps sum the sets in turn (warp
// q the sets q, q + kSetLanes, ..), the warps' sums are added in order and Finalize gets every
// particle's NV sums.  One thread per particle (finalize_kernel) walks the sets one after
// another: with tens of sets and a few thousand particles it waits for memory most of the time
// (FP64 adjoint of 1000 particles 80 -> 27 us with this pass and splits down to 64 sources).
#pragma once

#include "vpm_lanes.cuh"

namespace vpm {

constexpr int kSetLanes = 8;

// The splits of a one-sided sweep: every set holds target sums of every target.
struct SplitSets {
  int splits;
  __device__ __forceinline__ void ranges(int64_t, int& t, int& s) const {
    t = splits;
    s = 0;
  }
  template <int NV>
  __device__ __forceinline__ const double* source_set(const double* acc, int, int64_t,
                                                      int64_t&) const {
    return acc;
  }
};

// The values with source sums: the others' places in a source set are never written.
template <class Op>
struct SourceSums {
  __device__ __forceinline__ static constexpr bool has(int v) {
    return v < Op::kSymFrom && Op::carried(v);
  }
};
struct NoSourceSums {
  __device__ __forceinline__ static constexpr bool has(int) { return false; }
};

// Sets: for particle i, t sets of target sums (all NV values, acc[set][value][n]) and s sets of
// source sums (the values that Sources has) where source_set says, its values `stride` apart.
template <int NV, class Sources, class Sets, class Finalize>
__global__ void __launch_bounds__(32 * kSetLanes)
finalize_sets_kernel(const double* __restrict__ acc, const Sets sets, int64_t n,
                     const Finalize fin) {
  __shared__ double red[kSetLanes][NV][32];
  const int lane = threadIdx.x & 31, part = threadIdx.x >> 5;
  const int64_t i = int64_t(blockIdx.x) * 32 + lane;
  double v[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = 0.0;
  if (i < n) {
    int t, s;
    sets.ranges(i, t, s);
#pragma unroll 2
    for (int q = part; q < t; q += kSetLanes) {
      const double* p = acc + int64_t(q) * NV * n + i;
#pragma unroll
      for (int k = 0; k < NV; ++k) v[k] += p[int64_t(k) * n];
    }
#pragma unroll 2
    for (int q = part; q < s; q += kSetLanes) {
      int64_t stride = n;
      const double* p = sets.template source_set<NV>(acc, q, i, stride);
#pragma unroll
      for (int k = 0; k < NV; ++k)
        if (Sources::has(k)) v[k] += p[int64_t(k) * stride];
    }
  }
#pragma unroll
  for (int k = 0; k < NV; ++k) red[part][k][lane] = v[k];
  __syncthreads();
  if (part == 0 && i < n) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
#pragma unroll
      for (int q = 1; q < kSetLanes; ++q) v[k] += red[q][k][lane];
    }
    fin.write(v, i);
  }
}

}  // namespace vpm
