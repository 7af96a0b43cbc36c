// vpm_abi.cu -- C-ABI entry points, launch planning, pack and finalize kernels.  The
// library is one translation unit: the step and initial-condition kernels are included at
// the end.
//
// One pair-sum call = pack (reference AoS float64 -> packed records in the compute
// precision, inside the caller's workspace) -> tiled sweep (partials per source split,
// FP64) -> finalize (sum the splits in order, apply target-only factors, write the
// reference's output layout).  Scalars reduce the per-target values in a single block in a
// fixed order, so every result is deterministic.
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <unordered_map>
#include <utility>

#include <cuda.h>  // CUcontext / CUresult types only; no libcuda link

#include "vpm_b200.h"
#include "vpm_sweep.cuh"
#include "vpm_adjoint.cuh"
#include "vpm_rot.cuh"
#include "vpm_circle.cuh"
#include "vpm_triangle.cuh"
#include "vpm_sets.cuh"
#include "vpm_scalar.cuh"
#include "vpm_small.cuh"

namespace vpm {
namespace {

thread_local std::string g_last_error;

int fail(int code, const std::string& msg) {
  g_last_error = msg;
  return code;
}

int cuda_fail(cudaError_t e, const char* where) {
  return fail(VPM_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(e));
}

constexpr size_t kAlign = 256;
size_t align_up(size_t v) { return (v + kAlign - 1) / kAlign * kAlign; }

// ---- kernel configurations -----------------------------------------------------------
template <class T>
struct Cfg;
#ifndef VPM_FP32_R
#define VPM_FP32_R 4
#endif
#ifndef VPM_FP32_THREADS
#define VPM_FP32_THREADS 128
#endif
#ifndef VPM_FP32_MINB
#define VPM_FP32_MINB 1
#endif
// MINB: resident blocks per SM requested from the register allocator (launch bounds).
template <>
struct Cfg<float2> {
  static constexpr int R = VPM_FP32_R, THREADS = VPM_FP32_THREADS, TILE = 256, STAGES = 2,
                       MINB = VPM_FP32_MINB;
};
#ifndef VPM_FP64_R
#define VPM_FP64_R 1
#endif
#ifndef VPM_FP64_THREADS
#define VPM_FP64_THREADS 128
#endif
template <>
struct Cfg<double> {
  static constexpr int R = VPM_FP64_R, THREADS = VPM_FP64_THREADS, TILE = 128, STAGES = 2,
                       MINB = 1;
};

#ifndef VPM_MAX_SPLITS
#define VPM_MAX_SPLITS 64
#endif
constexpr int kMaxSplits = VPM_MAX_SPLITS;
// Shortest split of the sources.  Small sums are bound by the longest chain of sources a thread
// walks, and with the sets summed by several threads per particle (vpm_sets.cuh) a split more
// costs little: at 1000 particles chunks of 256 / 64 / 32 took 94 / 27 / 20 us for the FP64
// adjoint, 85 / 26 / 26 us for the FP64 and 42 / 22 / 24 us for the FP32c LES step sums.
template <class T>
constexpr int64_t kMinChunk = LaneTraits<T>::kLanes == 1 ? 32 : 64;
constexpr int64_t kMinChunkScalar = 256;  // of the scalar sums (Sweep::plan)
constexpr size_t kMaxPartialBytes = size_t(4) << 30;

struct Plan {
  int64_t tblocks = 0;
  int splits = 1;  // source splits; the both-sides sweep: its accumulator sets (2 per pair)
  int64_t chunk = 0;
  size_t smem = 0;
  int threads = 0;
  int r = 0;
  int nv = 0;
  int pairs = 0;  // both-sides sweep (vpm_rot.cuh): diagonal pairs per launch; 0 = one-sided
  // both-sides fused sum: 0 = built for VPM_ROT_MINB CTAs/SM, 1 = _ALT, 2 = 512-particle tiles
  int variant = 0;
  // both-sides sweep: the diagonal tiles run beside the (single) diagonal-pair launch on a
  // second stream, into their own accumulator sets after the pairs' ones
  int diag_beside = 0;
  // both-sides sweep over a triangle of tile pairs: its sets of target sums; 0 = no
  int triangle = 0;
  Shares shares{};  // of the one-launch schedules
  int circle = 0;  // FP64 both-sides sweep in one launch (vpm_circle.cuh)
  int small = 0;   // one launch from the caller's arrays (vpm_small.cuh); records: one-sided
  int scalar = 0;  // FP64 scalar diagnostics with each unordered pair once (vpm_scalar.cuh)
};

// What a plan's partial sums may take.
struct Budget {
  size_t one_sided, both_sides;
  bool compact;  // VPM_COMPACT_WORKSPACE: no triangle or circle, whose sets grow with n^2
  // bytes: the caller's limit.  Compact plans stay within 256 MB, but may use four sets of the
  // widest sums (18 values), the least the both-sides sweep works with.
  Budget(bool compact, size_t bytes, int64_t n)
      : one_sided(bytes), both_sides(bytes), compact(compact) {
    if (!compact) return;
    const size_t small = size_t(256) << 20, four = size_t(4 * 18 * 8) * size_t(n > 0 ? n : 0);
    one_sided = bytes < small ? bytes : small;
    const size_t both = small > four ? small : four;
    both_sides = bytes < both ? bytes : both;
  }
};

// FP32 self sums with at least this many particles evaluate each unordered pair once for both
// particles (vpm_set_symmetric_min_n changes it).  Measured crossover of the fused sum:
// one-sided 641 / 720 / 738 against both-sides 624 / 718 / 737 Gpairs/s at 16384 / 24576 /
// 32768 particles (velocity 1155 / 1258 / 1277 against 1160 / 1350 / 1419, PSE 1231 / 1344 /
// 1374 against 1380 / 1625 / 1728).
std::atomic<int64_t> g_sym_min_n{24576};

struct DevInfo {
  int sms = 0;
  int major = 0, minor = 0;
};

std::mutex g_mu;
std::unordered_map<int, DevInfo> g_dev;
std::map<std::pair<const void*, int>, int> g_occ;  // (kernel, device) -> resident blocks/SM

int device_info(DevInfo* out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  std::lock_guard<std::mutex> lk(g_mu);
  auto it = g_dev.find(dev);
  if (it == g_dev.end()) {
    DevInfo d;
    e = cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaDeviceGetAttribute(SM count)");
    cudaDeviceGetAttribute(&d.major, cudaDevAttrComputeCapabilityMajor, dev);
    cudaDeviceGetAttribute(&d.minor, cudaDevAttrComputeCapabilityMinor, dev);
    it = g_dev.emplace(dev, d).first;
  }
  *out = it->second;
  return VPM_OK;
}

int check_arch() {
  DevInfo d;
  int rc = device_info(&d);
  if (rc) return rc;
  if (d.major != 10 || d.minor != 0)
    return fail(VPM_ERR_ARCH, "libvpm_b200 is built for sm_100a (B200); current device is sm_" +
                                  std::to_string(d.major) + std::to_string(d.minor));
  return VPM_OK;
}

template <class Op, class T>
struct Sweep {
  using C = Cfg<T>;
  using RecT = typename Op::Record;
  static constexpr int NV = Op::NV;
  static constexpr int R = Op::kR ? Op::kR : C::R;
  // about the same tile bytes for every record width; FP32 tiles hold whole carry windows
  static constexpr int kTileRaw = int(C::TILE * sizeof(Rec<T>) / sizeof(RecT));
  static constexpr int TILE =
      LaneTraits<T>::kLanes == 2 ? kTileRaw / kCarryWindow * kCarryWindow : kTileRaw;
  static_assert(TILE >= kCarryWindow || LaneTraits<T>::kLanes == 1, "tile below a window");
  static constexpr size_t kSmem =
      sweep_smem_bytes<T, RecT, Op::NV, R, C::THREADS, TILE, C::STAGES>();
  static void* kernel() {
    return reinterpret_cast<void*>(&sweep_kernel<Op, T, R, C::THREADS, TILE, C::STAGES, C::MINB>);
  }

  // scalar: the sum's finalize is the one block of finalize_dot_kernel
  static int plan(int64_t m, int64_t n, Plan* p, size_t max_partial_bytes = kMaxPartialBytes,
                  bool scalar = false) {
    DevInfo d;
    int rc = device_info(&d);
    if (rc) return rc;
    int occ = 0;
    {
      // once per device: the shared-memory attribute, and the query that loads the kernel, so that
      // a stream capture after the plan only launches
      int dev = 0;
      cudaGetDevice(&dev);
      const auto key = std::make_pair(static_cast<const void*>(kernel()), dev);
      std::lock_guard<std::mutex> lk(g_mu);
      auto it = g_occ.find(key);
      if (it != g_occ.end()) {
        occ = it->second;
      } else {
        if (kSmem > 48 * 1024) {
          cudaError_t e = cudaFuncSetAttribute(kernel(), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               int(kSmem));
          if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(max dynamic smem)");
        }
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel(),
                                                                      C::THREADS, kSmem);
        if (e != cudaSuccess) return cuda_fail(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
        g_occ[key] = occ;
      }
    }
    if (occ < 1) occ = 1;
    const int64_t per_block = int64_t(C::THREADS) * R;
    p->tblocks = (m + per_block - 1) / per_block;
    p->smem = kSmem;
    p->threads = C::THREADS;
    p->r = R;
    p->nv = NV;
    p->splits = 1;
    p->chunk = n;
    if (n <= 0 || m <= 0) return VPM_OK;
    // Time of s splits, in units of one source for one block's targets on a busy SM: the blocks of
    // the busiest SM, two at a time at least (fewer do not keep its pipes full) and half a block
    // for the uneven end, each with a start and an end of about 40 sources, and the finalize's
    // pass over the sets at 5 TB/s.  Against the fill of whole waves of resident blocks, which
    // ignores that an SM with fewer blocks runs each faster (us): FP32c fused 623 -> 571 and
    // velocity 332 -> 306 at 20000, 862 -> 799 and 459 -> 429 at 24000, adjoint 2195 -> 2045;
    // probe vorticity of 10000 targets and sources in FP64 170 -> 158.  (Of 24, 40 and 12 sources,
    // 40 left no sum slower than the waves at 15 sizes from 4500 to 24400.)
    //
    // The scalar sums keep the waves and long splits: their finalize is one block that walks all
    // splits (FP32c kinetic energy 417 against 549 us at 20000, 45 against 74 at 4096).
    constexpr bool kFP32 = LaneTraits<T>::kLanes == 2;
    constexpr double kOps = (kFP32 ? 13.0 : 18.0) + 3.0 * NV;  // of a pair, about
    const double unit = double(C::THREADS) * R * kOps / (kFP32 ? 95.0 : 50.0);  // SM clocks
    const double set = double(m) * NV * 16.0 / 5e12 * 1.9e9 / unit;
    const int64_t min_chunk = scalar ? kMinChunkScalar : kMinChunk<T>;
    double best = -1.0;
    for (int s = 1; s <= kMaxSplits; ++s) {
      int64_t chunk = (n + s - 1) / s;
      chunk = (chunk + kCarryWindow - 1) / kCarryWindow * kCarryWindow;
      if (s > 1 && chunk < min_chunk) break;
      const int64_t se = (n + chunk - 1) / chunk;
      if (se != s) continue;
      if (size_t(se) * NV * size_t(m) * sizeof(double) > max_partial_bytes) break;
      const double total = double(p->tblocks) * double(se);
      double cost;
      if (scalar) {
        const double waves = total / (double(d.sms) * occ);
        cost = std::ceil(waves) / waves / (1.0 - 0.003 * double(se - 1));
      } else {
        const double blocks = std::ceil(total / d.sms);
        cost = (double(chunk) + 40.0) * ((blocks > 2.0 ? blocks : 2.0) + 0.5) + double(se) * set;
      }
      if (best < 0.0 || cost < best - 1e-12) {
        best = cost;
        p->splits = int(se);
        p->chunk = chunk;
      }
    }
    return VPM_OK;
  }

  static size_t partial_bytes(const Plan& p, int64_t m) {
    return size_t(p.splits) * NV * size_t(m) * sizeof(double);
  }

  static int launch(const Plan& p, const RecT* tgt, int64_t m, int64_t tgt_offset,
                    const RecT* src, int64_t n, double* partial, cudaStream_t st) {
    SweepArgs<RecT> a{tgt, m, tgt_offset, src, n, p.chunk, partial};
    dim3 grid(unsigned(p.tblocks), unsigned(p.splits));
    sweep_kernel<Op, T, R, C::THREADS, TILE, C::STAGES, C::MINB><<<grid, C::THREADS, p.smem, st>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "sweep launch");
    return VPM_OK;
  }
};

// ---- pack kernels ----------------------------------------------------------------------
__device__ __forceinline__ void set_elem(double& e, double v) { e = v; }
__device__ __forceinline__ void set_elem(float2& e, double v) {
  const float f = float(v);
  e = make_float2(f, f);
}

template <class E>
__global__ void pack_particles_kernel(const double* __restrict__ pos,
                                      const double* __restrict__ str,
                                      const double* __restrict__ rad,
                                      const double* __restrict__ nu, int64_t n,
                                      Rec<E>* __restrict__ out, int check_uniform) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (check_uniform && rad[i] != rad[0]) atomicOr(&g_device_errors, VPM_DEVERR_NONUNIFORM_CORE);
  Rec<E> r;
  set_elem(r.x, pos[3 * i]);
  set_elem(r.y, pos[3 * i + 1]);
  set_elem(r.z, pos[3 * i + 2]);
  set_elem(r.s, rad ? rad[i] : 0.0);
  set_elem(r.ax, str ? str[3 * i] : 0.0);
  set_elem(r.ay, str ? str[3 * i + 1] : 0.0);
  set_elem(r.az, str ? str[3 * i + 2] : 0.0);
  set_elem(r.nu, nu ? nu[i] : 0.0);
  out[i] = r;
}

template <class T>
int pack(const double* pos, const double* str, const double* rad, const double* nu, int64_t n,
         Rec<T>* out, cudaStream_t st, bool check_uniform = false) {
  if (n <= 0) return VPM_OK;
  const int threads = 256;
  const int64_t blocks = (n + threads - 1) / threads;
  pack_particles_kernel<T><<<unsigned(blocks), threads, 0, st>>>(pos, str, rad, nu, n, out,
                                                                 int(check_uniform && rad));
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "pack launch");
  return VPM_OK;
}

// ---- finalize kernels -----------------------------------------------------------------
// Splits from which the finalize of a one-sided sweep sums them with kSetLanes threads per
// particle (vpm_sets.cuh).
constexpr int kSetLanesMinSplits = 4;
constexpr int64_t kSetLanesMaxTargets = 1 << 16;

enum FinKind { FIN_VEL = 0, FIN_VORT = 1, FIN_STRETCH = 2, FIN_PSE = 3, FIN_VELSTRETCH = 4,
               FIN_LES = 5 };

template <int NV>
__device__ __forceinline__ void sum_splits(const double* __restrict__ part, int splits, int64_t m,
                                           int64_t i, double (&v)[NV]) {
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = 0.0;
  for (int s = 0; s < splits; ++s) {
    const double* p = part + int64_t(s) * NV * m;
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] += p[int64_t(k) * m + i];
  }
}

// The outputs of target i from its summed values v (KIND: which sums, which scaling).
template <class T, int KIND, int NV>
__device__ __forceinline__ void finalize_values(const double (&v)[NV], const Rec<T>* tgt,
                                                int64_t i, double* __restrict__ out,
                                                double* __restrict__ out2,
                                                double* __restrict__ out3) {
  if constexpr (KIND == FIN_VEL) {
    out[3 * i] = -v[0] * kOneOver4Pi;
    out[3 * i + 1] = -v[1] * kOneOver4Pi;
    out[3 * i + 2] = -v[2] * kOneOver4Pi;
  } else if constexpr (KIND == FIN_VORT) {
    const double c = 7.5 * kOneOver4Pi;
    out[3 * i] = v[0] * c;
    out[3 * i + 1] = v[1] * c;
    out[3 * i + 2] = v[2] * c;
  } else if constexpr (KIND == FIN_PSE) {
    const double c = 105.0 * elem(tgt[i].nu) * kOneOver4Pi;
    out[3 * i] = v[0] * c;
    out[3 * i + 1] = v[1] * c;
    out[3 * i + 2] = v[2] * c;
  } else {
    constexpr bool kVel = (KIND == FIN_VELSTRETCH || KIND == FIN_LES);
    constexpr int o = kVel ? 3 : 0;
    double* so = kVel ? out2 : out;
    const double bx = elem(tgt[i].ax), by = elem(tgt[i].ay), bz = elem(tgt[i].az);
    if constexpr (KIND == FIN_LES) {
      const double c = 7.5 * kOneOver4Pi;
      out3[3 * i] = v[9] * c;
      out3[3 * i + 1] = v[10] * c;
      out3[3 * i + 2] = v[11] * c;
    }
    if constexpr (kVel) {
      out[3 * i] = -v[0] * kOneOver4Pi;
      out[3 * i + 1] = -v[1] * kOneOver4Pi;
      out[3 * i + 2] = -v[2] * kOneOver4Pi;
    }
    const double Ax = v[o], Ay = v[o + 1], Az = v[o + 2];
    so[3 * i] = (by * Az - bz * Ay + 3.0 * v[o + 3]) * kOneOver4Pi;
    so[3 * i + 1] = (bz * Ax - bx * Az + 3.0 * v[o + 4]) * kOneOver4Pi;
    so[3 * i + 2] = (bx * Ay - by * Ax + 3.0 * v[o + 5]) * kOneOver4Pi;
  }
}

// Finalize of finalize_sets_kernel.  scalar (FIN_LES): particle i's enstrophy filter sum, from
// value 12 (both-sides sums) or from the three components E_i as a_i . E_i (one-sided sums).
template <class T, int KIND, int NV>
struct SetsFinalize {
  const Rec<T>* rec;
  double *out, *out2, *out3, *scalar;
  __device__ __forceinline__ void write(const double (&v)[NV], int64_t i) const {
    finalize_values<T, KIND, NV>(v, rec, i, out, out2, out3);
    if constexpr (KIND == FIN_LES) {
      if constexpr (NV == 13)
        scalar[i] = v[12];
      else
        scalar[i] = elem(rec[i].ax) * v[12] + elem(rec[i].ay) * v[13] + elem(rec[i].az) * v[14];
    }
  }
};

// One thread per particle; the sum over few splits, or of many particles.
template <int NV, class Finalize>
__global__ void finalize_kernel(const double* __restrict__ part, int splits, int64_t m,
                                const Finalize fin) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= m) return;
  double v[NV];
  sum_splits<NV>(part, splits, m, i, v);
  fin.write(v, i);
}

// part: [splits][NV][m]; fin.write(v, i) takes the sums of particle i.
template <int NV, class Finalize>
int finalize(const double* part, int splits, int64_t m, const Finalize& fin, cudaStream_t st) {
  if (m <= 0) return VPM_OK;
  if (splits >= kSetLanesMinSplits && m <= kSetLanesMaxTargets) {
    finalize_sets_kernel<NV, NoSourceSums, SplitSets><<<unsigned((m + 31) / 32), 32 * kSetLanes, 0, st>>>(
        part, SplitSets{splits}, m, fin);
  } else {
    const int threads = 256;
    finalize_kernel<NV>
        <<<unsigned((m + threads - 1) / threads), threads, 0, st>>>(part, splits, m, fin);
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? VPM_OK : cuda_fail(e, "finalize launch");
}

// Pair shards across GPUs: rows[i][v] = the sum over the sets s, in order, of acc[s][v][i].
// One particle's NV sums in a row, so each rank's target rows are one contiguous block for
// the reduce-scatter between the GPUs.
template <int NV>
__global__ void sets_to_rows_kernel(const double* __restrict__ acc, int sets, int64_t n,
                                    double* __restrict__ rows) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double v[NV];
  sum_splits<NV>(acc, sets, n, i, v);
#pragma unroll
  for (int k = 0; k < NV; ++k) rows[i * NV + k] = v[k];
}

// The outputs of targets [0, m) (records tgt) from their summed rows (m, NV).
template <class T, int KIND, int NV>
__global__ void finalize_rows_kernel(const double* __restrict__ rows, int64_t m,
                                     const Rec<T>* __restrict__ tgt, double* __restrict__ out,
                                     double* __restrict__ out2) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= m) return;
  double v[NV];
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = rows[i * NV + k];
  finalize_values<T, KIND, NV>(v, tgt, i, out, out2, nullptr);
}

constexpr int kReduceThreads = 1024;

// Single-block, fixed-order reduction of  scale * a_i . V_i  over all targets, V_i being their
// three sums.
template <class T>
__global__ void __launch_bounds__(kReduceThreads)
finalize_dot_kernel(const double* __restrict__ part, int splits, int64_t m,
                    const Rec<T>* __restrict__ tgt, double scale, double* __restrict__ out) {
  __shared__ double red[kReduceThreads];
  double acc = 0.0;
  for (int64_t i = threadIdx.x; i < m; i += kReduceThreads) {
    double v[3] = {0.0, 0.0, 0.0};
    for (int s = 0; s < splits; ++s) {
      const double* p = part + int64_t(s) * 3 * m;
#pragma unroll
      for (int k = 0; k < 3; ++k) v[k] += p[int64_t(k) * m + i];
    }
    acc += elem(tgt[i].ax) * v[0] + elem(tgt[i].ay) * v[1] + elem(tgt[i].az) * v[2];
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int w = kReduceThreads / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = red[0] * scale;
}

// scale * the sum of m values, in a fixed order (the same one as finalize_dot_kernel).
__global__ void __launch_bounds__(kReduceThreads)
finalize_sum_kernel(const double* __restrict__ v, int64_t m, double scale,
                    double* __restrict__ out) {
  __shared__ double red[kReduceThreads];
  double acc = 0.0;
#pragma unroll 8
  for (int64_t i = threadIdx.x; i < m; i += kReduceThreads) acc += v[i];
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int w = kReduceThreads / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = red[0] * scale;
}

__global__ void write_scalar_kernel(double* out, double v) { out[0] = v; }

template <class T, int KIND, int NV>
int finalize_vec(const double* part, int splits, int64_t m, const Rec<T>* tgt, double* out,
                 double* out2, cudaStream_t st, double* out3 = nullptr,
                 double* scalar = nullptr) {
  return finalize<NV>(part, splits, m, SetsFinalize<T, KIND, NV>{tgt, out, out2, out3, scalar},
                      st);
}

__global__ void zero_kernel(double* p, int64_t count) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < count) p[i] = 0.0;
}

int zero_out(double* p, int64_t count, cudaStream_t st) {
  if (count <= 0) return VPM_OK;
  zero_kernel<<<unsigned((count + 255) / 256), 256, 0, st>>>(p, count);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "zero launch");
  return VPM_OK;
}

// Both-sides sweep of an FP32 self sum (vpm_rot.cuh): launch 0 on the diagonal tiles, then
// ceil(floor(nt/2) / m) launches of m diagonal pairs each.
int current_context(void** ctx);

// A second stream per device and context for the both-sides sweep's diagonal tiles, with the
// two events that fork it from and join it to the caller's stream.  Created on first use
// with that context current (a stream belongs to one context, so another context, or the
// same device after a reset, gets its own); g_side_mu serialises the fork-launch-join
// sequence, so calls from several host threads never mix their events.
struct SideStream {
  cudaStream_t stream = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
};
std::mutex g_side_mu;
std::map<std::pair<int, void*>, SideStream> g_side;

// The calling thread holds g_side_mu.
int side_stream(SideStream** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  void* ctx = nullptr;
  int rc = current_context(&ctx);
  if (rc) return rc;
  const auto key = std::make_pair(dev, ctx);
  auto it = g_side.find(key);
  if (it == g_side.end()) {
    SideStream ss;
    e = cudaStreamCreateWithFlags(&ss.stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) return cuda_fail(e, "cudaStreamCreateWithFlags(side stream)");
    e = cudaEventCreateWithFlags(&ss.fork, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ss.join, cudaEventDisableTiming);
    if (e != cudaSuccess) return cuda_fail(e, "cudaEventCreateWithFlags(side stream)");
    it = g_side.emplace(key, ss).first;
  }
  *out = &it->second;
  return VPM_OK;
}

// Whether work of `st` can fork to the side stream.  It cannot while the side stream is part of
// another stream's capture, which a call made before that capture ends would join and break; such
// a call keeps its diagonal tiles on its own stream.  The calling thread holds g_side_mu.
bool side_free(const SideStream& ss, cudaStream_t st) {
  cudaStreamCaptureStatus side = cudaStreamCaptureStatusNone, own = side;
  unsigned long long side_id = 0, own_id = 0;
  cudaError_t e = cudaStreamGetCaptureInfo(ss.stream, &side, &side_id);
  if (e == cudaSuccess && side == cudaStreamCaptureStatusNone) return true;
  if (e == cudaSuccess) e = cudaStreamGetCaptureInfo(st, &own, &own_id);
  if (e != cudaSuccess) cudaGetLastError();
  return e == cudaSuccess && side == cudaStreamCaptureStatusActive && own == side &&
         own_id == side_id;
}

template <class Op>
struct RotSweep {
  static constexpr int NV = Op::NV;
  static constexpr int kMaxPairs = 32;
  static constexpr int kTile = rot_tile<Op>();
  static constexpr size_t kSmem = rot_smem_bytes<Op>();
  static int64_t tiles(int64_t n) { return (n + kTile - 1) / kTile; }
  static size_t set_bytes(int64_t n) { return size_t(NV) * size_t(n) * sizeof(double); }

  // Whether the planner takes this sweep for a self sum of n particles: the size threshold
  // (vpm_set_symmetric_min_n), two tiles at least, and the smallest set count (that of the
  // diagonal tiles' launch) within the caller's partial-sum budget.
  static bool usable(int64_t m, int64_t n, size_t max_partial_bytes) {
    return m == n && n >= g_sym_min_n.load() && tiles(n) >= 2 &&
           sets(1) * set_bytes(n) <= max_partial_bytes;
  }
  // accumulator sets of a plan with m diagonal pairs per launch: 2 per pair, and at least the
  // kRotDiagSplit the diagonal tiles' launch writes (after the pairs' sets when it runs beside
  // the pair launches)
  static int64_t sets(int m, bool beside = false) {
    if (beside) return 2 * int64_t(m) + kRotDiagSplit;
    return 2 * m > kRotDiagSplit ? 2 * m : kRotDiagSplit;
  }

  // The kernel of the operator's precision: rot_sweep_kernel (FP32 lanes) or
  // rot64_sweep_kernel (FP64).
  template <bool DIAG>
  static const void* kernel_ptr() {
    if constexpr (Op::kFP64)
      return reinterpret_cast<const void*>(&rot64_sweep_kernel<Op, DIAG>);
    else
      return reinterpret_cast<const void*>(&rot_sweep_kernel<Op, DIAG>);
  }
  template <bool DIAG>
  static void launch_kernel(unsigned grid, const RotArgs& a, cudaStream_t st) {
    if constexpr (Op::kFP64)
      rot64_sweep_kernel<Op, DIAG><<<grid, kRotThreads, kSmem, st>>>(a);
    else
      rot_sweep_kernel<Op, DIAG><<<grid, kRotThreads, kSmem, st>>>(a);
  }

  // Shared-memory attributes and resident CTAs per SM, once per device (cached like the
  // one-sided sweeps' plans).
  static int prepare(int* occ) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    const void* ks = kernel_ptr<false>();
    const void* kd = kernel_ptr<true>();
    const auto key = std::make_pair(ks, dev);
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_occ.find(key);
    if (it != g_occ.end()) {
      *occ = it->second;
      return VPM_OK;
    }
    for (const void* fn : {kd, ks}) {
      e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmem));
      if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(both-sides sweep)");
    }
    int o = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, ks, kRotThreads, kSmem);
    if (e != cudaSuccess) return cuda_fail(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
    *occ = o > 0 ? o : 1;
    g_occ[key] = *occ;
    return VPM_OK;
  }

  // Waves (rounds of resident CTAs, each about one tile pair long) that the diagonal-pair
  // launches of a plan with m pairs per launch take: npairs / m launches of m nt CTAs and a
  // last one of the remaining pairs.
  static int64_t pair_waves(int64_t npairs, int64_t nt, int64_t m, int64_t slots) {
    const int64_t full = npairs / m, rem = npairs - full * m;
    return full * ((m * nt + slots - 1) / slots) + (rem * nt + slots - 1) / slots;
  }

  // Creates the side stream now, outside any stream capture of the launch that follows.
  static int prepare_side() {
    std::lock_guard<std::mutex> lk(g_side_mu);
    SideStream* ss = nullptr;
    return side_stream(&ss);
  }

  // eff_out: the fraction of whole waves the chosen launches fill (ideal waves / waves)
  static int plan(int64_t n, Plan* p, size_t max_partial_bytes, double* eff_out = nullptr) {
    DevInfo d;
    int rc = device_info(&d);
    if (rc) return rc;
    int occ = 1;
    rc = prepare(&occ);
    if (rc) return rc;
    const int64_t nt = tiles(n);
    const int64_t npairs = nt / 2;
    const int64_t slots = int64_t(d.sms) * occ;
    // Pairs per launch, two candidates within the caller's workspace budget: m0, the first m
    // whose own launch fills 97 % of whole waves (else the best such fill), and m1, the m whose
    // launches take the fewest waves in all (the smaller m on a tie).  m0 is kept unless m1
    // saves more than 1 % of the waves: at equal wave counts the launches of m0 measured up to
    // 5 % faster (fused sum at 65536, LES sums at 262144), while m1 gains 1.5 % at 2^20 and 7 %
    // at 49152.  (Splitting each tile pair's sources over several CTAs, to fill the waves at
    // small n, measured slower: every part repeats the target side's carries and final FP64
    // atomics, and the sets to zero and sum multiply.)
    int m0 = 1;
    double be = -1.0;
    for (int m = 1; m <= kMaxPairs && m <= npairs; ++m) {
      if (m > 1 && sets(m) * set_bytes(n) > max_partial_bytes) break;
      const double waves = double(m) * nt / double(slots);
      const double eff = waves / std::ceil(waves);
      if (eff > be + 1e-9) {
        be = eff;
        m0 = m;
      }
      if (eff >= 0.97) break;
    }
    int m1 = 1;
    int64_t w1 = pair_waves(npairs, nt, 1, slots);
    for (int m = 2; m <= kMaxPairs && m <= npairs; ++m) {
      if (sets(m) * set_bytes(n) > max_partial_bytes) break;
      const int64_t w = pair_waves(npairs, nt, m, slots);
      if (w < w1) {
        w1 = w;
        m1 = m;
      }
    }
    const int64_t w0 = pair_waves(npairs, nt, m0, slots);
    const bool keep0 = double(w0) <= 1.01 * double(w1);
    const int best_m = keep0 ? m0 : m1;
    const int64_t best_w = keep0 ? w0 : w1;
    const double best = double(npairs) * nt / double(slots) / double(best_w);
    if (eff_out) *eff_out = best;
    // Small n (pair launches of at most 64 waves of whole tile pairs): the diagonal tiles' CTAs
    // (a quarter tile of sources each) run beside the pair launches on a second stream, into
    // four sets of their own, and take the slots their waves leave free, instead of a launch
    // of their own before them.  Measured (Gpairs/s, own launch -> beside): fused sum 574 ->
    // 622 at 16384, 739 -> 748 at 32768; velocity 1427 -> 1477 and PSE 1733 -> 1808 at 32768;
    // 1-2 % at 49152.  At large n that launch is a few tenths of a percent of the sweep.
    const bool beside = best_w <= 64 && sets(best_m, true) * set_bytes(n) <= max_partial_bytes;
    if (beside) {
      rc = prepare_side();
      if (rc) return rc;
    }
    p->diag_beside = beside ? 1 : 0;
    p->pairs = best_m;
    p->tblocks = nt;
    p->splits = int(sets(best_m, beside));
    p->chunk = n;
    p->smem = kSmem;
    p->threads = kRotThreads;
    p->r = 2 * Op::kP;
    p->nv = NV;
    return VPM_OK;
  }

  // acc: [p.splits][NV][n] FP64, zeroed here.
  static int launch(const Plan& p, const void* rec, int64_t n, double* acc,
                    cudaStream_t st) {
    const int nt = int(tiles(n));
    int occ = 1;
    int rc = prepare(&occ);
    if (!rc) rc = zero_out(acc, int64_t(p.splits) * NV * n, st);
    if (rc) return rc;
    cudaError_t e = cudaSuccess;
    const int npairs = nt / 2;
    SideStream* ss = nullptr;
    std::unique_lock<std::mutex> lk(g_side_mu, std::defer_lock);
    bool beside = false;
    if (p.diag_beside) {
      // the pair launches on the caller's stream, the diagonal tiles on the side stream into
      // sets [sets of the pairs, + kRotDiagSplit); the caller's stream waits for both (fork
      // and join by events, so CUDA-graph capture records the same dependencies)
      lk.lock();
      rc = side_stream(&ss);
      if (rc) return rc;
      beside = side_free(*ss, st);
      if (beside) e = cudaEventRecord(ss->fork, st);
      if (e != cudaSuccess) return cuda_fail(e, "cudaEventRecord(fork)");
    } else {
      launch_kernel<true>(unsigned(nt * kRotDiagSplit), RotArgs{rec, n, nt, 0, acc}, st);
      e = cudaGetLastError();
      if (e != cudaSuccess) return cuda_fail(e, "both-sides sweep launch");
    }
    for (int k0 = 1; k0 <= npairs; k0 += p.pairs) {
      const int m = (npairs - k0 + 1 < p.pairs) ? npairs - k0 + 1 : p.pairs;
      launch_kernel<false>(unsigned(m * nt), RotArgs{rec, n, nt, k0, acc}, st);
      e = cudaGetLastError();
      if (e != cudaSuccess) return cuda_fail(e, "both-sides sweep launch");
    }
    if (p.diag_beside) {
      if (beside) e = cudaStreamWaitEvent(ss->stream, ss->fork, 0);
      if (e != cudaSuccess) return cuda_fail(e, "cudaStreamWaitEvent(fork)");
      RotArgs d{rec, n, nt, 0, acc};
      d.set0 = 2 * p.pairs;
      launch_kernel<true>(unsigned(nt * kRotDiagSplit), d, beside ? ss->stream : st);
      e = cudaGetLastError();
      if (e != cudaSuccess) return cuda_fail(e, "both-sides sweep launch");
      if (!beside) return VPM_OK;
      e = cudaEventRecord(ss->join, ss->stream);
      if (e != cudaSuccess) return cuda_fail(e, "cudaEventRecord(join)");
      e = cudaStreamWaitEvent(st, ss->join, 0);
      if (e != cudaSuccess) return cuda_fail(e, "cudaStreamWaitEvent(join)");
    }
    return VPM_OK;
  }

  // Part of a sweep (pair shards across GPUs): the diagonal tiles [t_begin, t_end) and the
  // diagonal pairs k in [k_begin, k_end) (k = 1 .. nt / 2), in launches of p.pairs pairs, on
  // the caller's stream into the sets of a plan without the side stream.
  // acc: [sets(p.pairs)][NV][n] FP64, zeroed here.
  static int launch_part(const Plan& p, const void* rec, int64_t n, double* acc, int t_begin,
                         int t_end, int k_begin, int k_end, cudaStream_t st) {
    const int nt = int(tiles(n));
    int occ = 1;
    int rc = prepare(&occ);
    if (!rc) rc = zero_out(acc, sets(p.pairs) * NV * n, st);
    if (rc) return rc;
    cudaError_t e = cudaSuccess;
    if (t_end > t_begin) {
      RotArgs d{rec, n, nt, 0, acc};
      d.tile0 = t_begin;
      launch_kernel<true>(unsigned((t_end - t_begin) * kRotDiagSplit), d, st);
      e = cudaGetLastError();
      if (e != cudaSuccess) return cuda_fail(e, "both-sides sweep launch");
    }
    for (int k0 = k_begin; k0 < k_end; k0 += p.pairs) {
      const int m = (k_end - k0 < p.pairs) ? k_end - k0 : p.pairs;
      launch_kernel<false>(unsigned(m * nt), RotArgs{rec, n, nt, k0, acc}, st);
      e = cudaGetLastError();
      if (e != cudaSuccess) return cuda_fail(e, "both-sides sweep launch");
    }
    return VPM_OK;
  }
};

// FP64 scalar diagnostics over all particles (vpm_scalar.cuh): launch plan and launches.
template <class Op>
struct ScalarSweep {
  template <int R>
  static const void* kernel() {
    return reinterpret_cast<const void*>(&scalar_pairs_kernel<Op, R>);
  }

  template <int R>
  static int occupancy(int* occ) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    const auto key = std::make_pair(kernel<R>(), dev);
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_occ.find(key);
    if (it == g_occ.end()) {
      int o = 0;
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, kernel<R>(), kScalarThreads, 0);
      if (e != cudaSuccess) return cuda_fail(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
      it = g_occ.emplace(key, o > 0 ? o : 1).first;
    }
    *occ = it->second;
    return VPM_OK;
  }

  // Splits of a target tile's source list: the count whose waves of equal blocks take the least
  // time, a block costing its pieces and about one more for its start and reduction.
  template <int R>
  static double best_splits(int64_t n, int64_t slots, Plan* p) {
    const int64_t T = int64_t(kScalarThreads) * R;
    const int64_t nt = (n + T - 1) / T;
    const int64_t pieces = (1 + nt / 2) * (T / kScalarPiece);
    double best = -1.0;
    for (int64_t s = 1; s <= 256 && s <= pieces; ++s) {
      const int64_t chunk = (pieces + s - 1) / s;
      const int64_t se = (pieces + chunk - 1) / chunk;
      if (se != s) continue;
      const double waves = std::ceil(double(nt * se) / double(slots));
      const double cost = waves * (double(chunk) + 1.0) * R;
      if (best < 0.0 || cost < best) {
        best = cost;
        p->splits = int(se);
        p->chunk = chunk;
      }
    }
    p->tblocks = nt;
    p->threads = kScalarThreads;
    p->r = R;
    p->nv = 1;
    p->scalar = 1;
    return best;
  }

  static int plan(int64_t n, Plan* p) {
    DevInfo d;
    int rc = device_info(&d);
    int o1 = 1, o2 = 1;
    if (!rc) rc = occupancy<1>(&o1);
    if (!rc) rc = occupancy<2>(&o2);
    if (rc) return rc;
    Plan p1, p2;
    // work per SM and piece is R x the resident blocks; the cheaper of the two builds
    const double c1 = best_splits<1>(n, int64_t(d.sms) * o1, &p1) * o1;
    const double c2 = best_splits<2>(n, int64_t(d.sms) * o2, &p2) * o2;
    *p = c1 < c2 ? p1 : p2;
    return VPM_OK;
  }

  // doubles of partial sums: [p.splits][p.tblocks][2] (the same for every operator)
  static size_t partials(const Plan& p) { return size_t(p.splits) * size_t(p.tblocks) * 2; }

  // partial: partials(p) doubles
  static int launch(const Plan& p, const Rec<double>* rec, int64_t n, double* partial,
                    double scale, double* out, cudaStream_t st) {
    const ScalarArgs a{rec, n, int(p.tblocks), int(p.chunk), partial};
    const dim3 grid(unsigned(p.tblocks), unsigned(p.splits));
    if (p.r == 1)
      scalar_pairs_kernel<Op, 1><<<grid, kScalarThreads, 0, st>>>(a);
    else
      scalar_pairs_kernel<Op, 2><<<grid, kScalarThreads, 0, st>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "scalar sweep launch");
    // each unordered pair was counted once
    scalar_total_kernel<<<1, 1024, 0, st>>>(partial, int(p.tblocks) * p.splits, 2.0 * scale, out);
    e = cudaGetLastError();
    return e == cudaSuccess ? VPM_OK : cuda_fail(e, "reduce launch");
  }
};

// ---- adjoint: pack, finalize --------------------------------------------------------------
template <class E>
__global__ void pack_grad_kernel(const double* __restrict__ pos, const double* __restrict__ str,
                                 const double* __restrict__ rad, const double* __restrict__ nu,
                                 const double* __restrict__ gu, const double* __restrict__ gs,
                                 int64_t n, RecG<E>* __restrict__ out) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  RecG<E> r;
  set_elem(r.x, pos[3 * i]);
  set_elem(r.y, pos[3 * i + 1]);
  set_elem(r.z, pos[3 * i + 2]);
  set_elem(r.s, rad[i]);
  set_elem(r.ax, str[3 * i]);
  set_elem(r.ay, str[3 * i + 1]);
  set_elem(r.az, str[3 * i + 2]);
  set_elem(r.nu, nu ? 105.0 * nu[i] : 0.0);
  set_elem(r.ux, -kOneOver4Pi * gu[3 * i]);
  set_elem(r.uy, -kOneOver4Pi * gu[3 * i + 1]);
  set_elem(r.uz, -kOneOver4Pi * gu[3 * i + 2]);
  const double ax = str[3 * i], ay = str[3 * i + 1], az = str[3 * i + 2];
  const double sx = kOneOver4Pi * gs[3 * i], sy = kOneOver4Pi * gs[3 * i + 1],
               sz = kOneOver4Pi * gs[3 * i + 2];
  set_elem(r.gx, sx);
  set_elem(r.gy, sy);
  set_elem(r.gz, sz);
  set_elem(r.mx, ay * sz - az * sy);  // m = a x s'
  set_elem(r.my, az * sx - ax * sz);
  set_elem(r.mz, ax * sy - ay * sx);
  set_elem(r.pad0, 0.0);
  set_elem(r.pad1, 0.0);
  set_elem(r.pad2, 0.0);
  out[i] = r;
}

// The gradients of particle i from its summed values v.
template <class E, int NV, bool PSE>
__device__ __forceinline__ void finalize_vjp_values(const double (&v)[NV],
                                                    const RecG<E>* __restrict__ tgt, int64_t i,
                                                    double* __restrict__ gx,
                                                    double* __restrict__ ga,
                                                    double* __restrict__ gsig,
                                                    double* __restrict__ gnu) {
  const RecG<E>& t = tgt[i];
  const double ax = elem(t.ax), ay = elem(t.ay), az = elem(t.az);
  const double ux = elem(t.ux), uy = elem(t.uy), uz = elem(t.uz);
  const double sx = elem(t.gx), sy = elem(t.gy), sz = elem(t.gz);
  const double Gx = v[VJ_GA], Gy = v[VJ_GA + 1], Gz = v[VJ_GA + 2];
  const double Hx = v[VJ_GU], Hy = v[VJ_GU + 1], Hz = v[VJ_GU + 2];
  // xbar += G_a x u'_k - a_k x G_u
  gx[3 * i] = v[VJ_X] + (Gy * uz - Gz * uy) - (ay * Hz - az * Hy);
  gx[3 * i + 1] = v[VJ_X + 1] + (Gz * ux - Gx * uz) - (az * Hx - ax * Hz);
  gx[3 * i + 2] = v[VJ_X + 2] + (Gx * uy - Gy * ux) - (ax * Hy - ay * Hx);
  // abar += G_a x s'_k  (+ PSE: sum k nu'_l s'_l - (sum k) nu'_k s'_k)
  double bx = v[VJ_A] + (Gy * sz - Gz * sy);
  double by = v[VJ_A + 1] + (Gz * sx - Gx * sz);
  double bz = v[VJ_A + 2] + (Gx * sy - Gy * sx);
  if constexpr (PSE) {
    const double kn = v[VJ_K] * elem(t.nu);
    bx += v[VJ_KS] - kn * sx;
    by += v[VJ_KS + 1] - kn * sy;
    bz += v[VJ_KS + 2] - kn * sz;
  }
  ga[3 * i] = bx;
  ga[3 * i + 1] = by;
  ga[3 * i + 2] = bz;
  gsig[i] = 0.5 * v[VJ_S];
  if (gnu) gnu[i] = PSE ? 105.0 * v[VJ_NU] : 0.0;
}

template <class E, bool PSE>
struct SetsFinalizeVjp {
  const RecG<E>* rec;
  double *gx, *ga, *gs, *gnu;
  static constexpr int NV = OpRhsVjp<E, false, PSE>::NV;
  __device__ __forceinline__ void write(const double (&v)[NV], int64_t i) const {
    finalize_vjp_values<E, NV, PSE>(v, rec, i, gx, ga, gs, gnu);
  }
};

// Gradients of the kinetic energy (OpKeGrad's seven sums).
struct SetsFinalizeKeGrad {
  double *gx, *ga, *gs;
  __device__ __forceinline__ void write(const double (&v)[7], int64_t i) const {
    const double c = 2.0 / (16.0 * kPi);
    gx[3 * i] = c * v[0];
    gx[3 * i + 1] = c * v[1];
    gx[3 * i + 2] = c * v[2];
    ga[3 * i] = c * v[3];
    ga[3 * i + 1] = c * v[4];
    ga[3 * i + 2] = c * v[5];
    gs[i] = 0.5 * c * v[6];
  }
};

// ---- both-sides sweep over a triangle of tile pairs (vpm_triangle.cuh, vpm_circle.cuh) --------
// Its partial sums may take this much; past it the sweep is the many-launch one (vpm_rot.cuh),
// whose accumulators do not grow with n^2.  In FP32c the many-launch sweep's waves are long enough
// from about 150000 particles for the velocity with general cores (ms, many launches / triangle):
// 12.16 / 12.12 at 149999, 13.77 / 13.80 at 160000, 17.30 / 17.43 at 180001, 24.58 / 24.79 at 215000.
// Above that the others are within 1 % either way but for the fused sum at 160000 (26.33 / 25.83,
// with one core 25.13 / 24.58; 32.62 / 32.68 at 180001) and the velocity with one core (12.47 / 12.26
// at 160000, 19.37 / 19.11 at 200000).  LES sums and adjoints are past the 2 GB before 150000 (from
// about 135000, 129000 and with PSE 83000), the fused sum from about 197000.
constexpr size_t kMaxTriangleBytes = size_t(2) << 30;
constexpr int64_t kMaxTriangleN32 = 150000;

template <class Op>
struct TriSweep {
  static constexpr int NV = Op::NV;
  static constexpr int kTile = rot_tile<Op>();
  static constexpr int kUnit = Op::kFP64 ? 32 : kTriUnit;
  static constexpr size_t smem() {
    if constexpr (Op::kFP64)
      return lists64_smem_bytes<Op>();
    else
      return rot_smem_bytes<Op>();
  }
  static constexpr size_t kSmem = smem();

  static const void* kernel_ptr() {
    if constexpr (Op::kFP64)
      return reinterpret_cast<const void*>(&rot64_lists_kernel<Op, TriLists64>);
    else
      return reinterpret_cast<const void*>(&rot_triangle_kernel<Op>);
  }

  static int prepare(int* occ) {
    const void* fn = kernel_ptr();
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    const auto key = std::make_pair(fn, dev);
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_occ.find(key);
    if (it == g_occ.end()) {
      e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmem));
      if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(triangle sweep)");
      int o = 0;
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, fn, kRotThreads, kSmem);
      if (e != cudaSuccess) return cuda_fail(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
      it = g_occ.emplace(key, o > 0 ? o : 1).first;
    }
    *occ = it->second;
    return VPM_OK;
  }

  // p: the many-launch plan of the same build.  Sets p->triangle and p->splits where the partial
  // sums fit; the other fields stay (the pair shards across GPUs use them).
  static int plan(int64_t n, Plan* p, size_t max_partial_bytes) {
    DevInfo d;
    int occ = 1;
    int rc = device_info(&d);
    if (!rc) rc = prepare(&occ);
    if (!rc) rc = RotSweep<Op>::prepare_side();
    if (rc || n >= (int64_t(1) << 30) || (!Op::kFP64 && n > kMaxTriangleN32)) return rc;
    const TriLists l(n, kTile, kUnit);
    if (size_t(l.nt / 2) * NV * size_t(n) * sizeof(double) > kMaxTriangleBytes) return VPM_OK;
    const Shares shares = Shares::make(l.total(), int64_t(d.sms) * occ);
    const int tsets = target_sets(l, shares);
    const int64_t sets =
        kRotDiagSplit + tsets + (l.before(l.nt - 1, n, kTile) + n - 1) / n;
    const size_t bytes = size_t(sets) * NV * size_t(n) * sizeof(double);
    if (bytes > max_partial_bytes || bytes > kMaxTriangleBytes) return VPM_OK;
    p->triangle = tsets;
    p->shares = shares;
    p->splits = int(sets);
    return VPM_OK;
  }

  // acc: [p.splits][NV][n]: the diagonal tiles' sets, the target sets, the source sets.  The
  // diagonal tiles run beside on the side stream, launched first, so that their few blocks are
  // done when the shares that wait for their places begin.
  template <class Finalize>
  static int launch(const Plan& p, const void* rec, int64_t n, double* acc, const Finalize& fin,
                    cudaStream_t st) {
    const TriLists l(n, kTile, kUnit);
    const int tsets = p.triangle;
    double* target = acc + int64_t(kRotDiagSplit) * NV * n;
    double* source = target + int64_t(tsets) * NV * n;
    int rc = zero_out(acc, int64_t(kRotDiagSplit) * NV * n, st);
    if (!rc) {
      std::unique_lock<std::mutex> lk(g_side_mu);
      SideStream* ss = nullptr;
      rc = side_stream(&ss);
      if (rc) return rc;
      const bool beside = side_free(*ss, st);
      cudaError_t e = cudaSuccess;
      if (beside) e = cudaEventRecord(ss->fork, st);
      if (beside && e == cudaSuccess) e = cudaStreamWaitEvent(ss->stream, ss->fork, 0);
      if (e != cudaSuccess) return cuda_fail(e, "side stream fork");
      RotSweep<Op>::template launch_kernel<true>(unsigned(l.nt * kRotDiagSplit),
                                                 RotArgs{rec, n, l.nt, 0, acc},
                                                 beside ? ss->stream : st);
      e = cudaGetLastError();
      if (e != cudaSuccess) return cuda_fail(e, "both-sides sweep launch");
      const unsigned grid = unsigned(p.shares.blocks());
      if constexpr (Op::kFP64) {
        const Sweep64Args a{rec, int(n), p.shares, target, source};
        rot64_lists_kernel<Op, TriLists64><<<grid, kRotThreads, kSmem, st>>>(a);
      } else {
        const TriArgs a{rec, int(n), l.nt, p.shares, target, source};
        rot_triangle_kernel<Op><<<grid, kRotThreads, kSmem, st>>>(a);
      }
      e = cudaGetLastError();
      if (e != cudaSuccess) return cuda_fail(e, "triangle sweep launch");
      if (beside) e = cudaEventRecord(ss->join, ss->stream);
      if (beside && e == cudaSuccess) e = cudaStreamWaitEvent(st, ss->join, 0);
      if (e != cudaSuccess) return cuda_fail(e, "side stream join");
    }
    if (rc) return rc;
    const TriSets sets{l, p.shares, kTile, kRotDiagSplit, n, source};
    finalize_sets_kernel<NV, SourceSums<Op>, TriSets, Finalize>
        <<<unsigned((n + 31) / 32), 32 * kSetLanes, 0, st>>>(acc, sets, n, fin);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? VPM_OK : cuda_fail(e, "finalize launch");
  }
};

// ---- FP64 both-sides sweep in one launch (vpm_circle.cuh) ------------------------------------
// Lower end of its range, a sixth of the both-sides threshold (so that vpm_set_symmetric_min_n
// moves both): 4096 particles by default.  Measured against the one-sided sweeps (us, velocity /
// fused / stretching / PSE / LES / adjoint): 36 / 58 / 43 / 31 / 73 / 90 against 26 / 39 / 35 / 27
// / 73 / 80 at 3072, 37 / 61 / 44 / 32 / 92 / 115 against 39 / 64 / 59 / 39 / 106 / 149 at 4096,
// 50 / 82 / 61 / 43 / 134 / 167 against 61 / 92 / 85 / 57 / 150 / 219 at 5000.
int64_t circle_min_n() { return g_sym_min_n.load() / 6; }

template <class Op>
struct CircleSweep {
  static constexpr int NV = Op::NV;
  static constexpr int kTile = rot_tile<Op>();
  static constexpr size_t kSmem = lists64_smem_bytes<Op>();

  static int prepare(int* occ) {
    const void* fn = reinterpret_cast<const void*>(&rot64_lists_kernel<Op, CircleLists>);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    const auto key = std::make_pair(fn, dev);
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_occ.find(key);
    if (it == g_occ.end()) {
      e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmem));
      if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute(circle sweep)");
      int o = 0;
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, fn, kRotThreads, kSmem);
      if (e != cudaSuccess) return cuda_fail(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
      it = g_occ.emplace(key, o > 0 ? o : 1).first;
    }
    *occ = it->second;
    return VPM_OK;
  }

  // Fills the plan; leaves p->circle 0 where the sets exceed the budget.
  static int plan(int64_t n, Plan* p, size_t max_partial_bytes) {
    DevInfo d;
    int occ = 1;
    int rc = device_info(&d);
    if (!rc) rc = prepare(&occ);
    if (rc) return rc;
    const CircleLists l(n, kTile);
    // (the source sets alone: no count of the target sets at sizes that are far past the budget)
    if (size_t(l.half) * NV * size_t(n) * sizeof(double) > max_partial_bytes) return VPM_OK;
    p->shares = Shares::make(l.total(), int64_t(d.sms) * occ);
    const int64_t sets = target_sets(l, p->shares) + l.half;
    if (size_t(sets) * NV * size_t(n) * sizeof(double) > max_partial_bytes) return VPM_OK;
    p->circle = 1;
    p->tblocks = l.nt;
    p->splits = int(sets);
    p->chunk = n;
    p->smem = kSmem;
    p->threads = kRotThreads;
    p->r = 2 * Op::kP;
    p->nv = NV;
    return VPM_OK;
  }

  // acc: [p.splits][NV][n]; fin.write(v, i) takes the sums of particle i.
  template <class Finalize>
  static int launch(const Plan& p, const void* rec, int64_t n, double* acc, const Finalize& fin,
                    cudaStream_t st) {
    const CircleLists l(n, kTile);
    const int tsets = p.splits - l.half;
    const Sweep64Args a{rec, int(n), p.shares, acc, acc + int64_t(tsets) * NV * n};
    rot64_lists_kernel<Op, CircleLists>
        <<<unsigned(p.shares.blocks()), kRotThreads, kSmem, st>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "circle sweep launch");
    const CircleSets sets{l, p.shares, kTile, tsets, n};
    finalize_sets_kernel<NV, SourceSums<Op>, CircleSets, Finalize>
        <<<unsigned((n + 31) / 32), 32 * kSetLanes, 0, st>>>(acc, sets, n, fin);
    e = cudaGetLastError();
    return e == cudaSuccess ? VPM_OK : cuda_fail(e, "finalize launch");
  }
};


// The FP64 plan of a self sum of n particles on the both-sides schedules, if it takes one
// (p->circle or p->pairs set).  MULTI: from the threshold on the sum takes the triangle, and the
// many-launch sweep past the triangle's budget; otherwise the circle at all sizes its sets fit.
template <class Op, bool MULTI>
int plan_both64(int64_t m, int64_t n, Plan* p, const Budget& b) {
  if (m != n) return VPM_OK;
  const size_t mpb = b.both_sides;
  const bool large = RotSweep<Op>::usable(m, n, mpb);
  if (!b.compact && n > 0 && n >= circle_min_n() && n < (int64_t(1) << 30) &&
      RotSweep<Op>::tiles(n) >= 2 && !(MULTI && n >= g_sym_min_n.load())) {
    int rc = CircleSweep<Op>::plan(n, p, mpb);
    if (rc || p->circle) return rc;
  }
  if (!large) return VPM_OK;
  int rc = RotSweep<Op>::plan(n, p, mpb);
  if constexpr (MULTI) {
    if (!rc && !b.compact) rc = TriSweep<Op>::plan(n, p, mpb);
  }
  return rc;
}

// The FP32 both-sides plan of a self sum: the many-launch sweep's, and the one-launch form where
// its partial sums fit.
template <class Op>
int plan_both32(int64_t n, Plan* p, const Budget& b) {
  int rc = RotSweep<Op>::plan(n, p, b.both_sides);
  if (!rc && !b.compact) rc = TriSweep<Op>::plan(n, p, b.both_sides);
  return rc;
}

// ---- small sums in one launch (vpm_small.cuh) ---------------------------------------------
// Taken for a vector sum from the caller's arrays with fewer than kSmallSources sources (four
// windows per warp of the largest cluster) and at most small_pairs pairs.  Measured against the
// three launches (us, self sums): FP64 velocity 15.0 / 27 at 2000 and 28.2 / 26.1 at 3000
// particles, fused 20.2 / 37 and 39.6 / 39.1; FP32c velocity 9.1 / 24 at 2000, 14.8 / 16.8 at 3000
// and 22.3 / 25.3 at 4000, fused 13.5 / 45, 22.0 / 29.4 and 34.7 / 41.1.
constexpr int64_t kSmallSources = 4096;
template <class T>
constexpr int64_t small_pairs = LaneTraits<T>::kLanes == 1 ? 6000000 : 16000000;
// Most blocks of targets (32 per lane).  Past it the limit on pairs leaves fewer than 62 sources:
// one or two windows for the four warps of a block, the others idle.  Probe sums, us, three
// launches / one (velocity, vorticity): FP64 131072 x 40 21.9 / 25.9 and 20.3 / 26.2, 300000 x 10
// 21.3 / 31.8 and 20.3 / 32.0, 10^6 x 1 38.9 / 75.0; FP32c 300000 x 40 25.8 / 28.5 and 24.0 / 26.3,
// 10^6 x 16 48.2 / 65.2.  Below it, FP64 62000 x 96 25.4 / 19.9, 50000 x 10 9.4 / 8.0, 10000 x 300
// 34.2 / 17.0, 3000 x 2000 35.1 / 21.8; FP32c 250000 x 64 31.1 / 27.5, 100000 x 40 15.0 / 12.7,
// 8000 x 2000 28.9 / 24.0.  (FP64 at 100000 targets and 1 to 40 sources: 9.4 to 19.8 / 9.8 to 20.5
// on the device, and 29 / 14 to 23 for a call that is not captured.)
template <class T>
constexpr int64_t kSmallBlocks = LaneTraits<T>::kLanes == 1 ? 3200 : 4096;

int64_t small_windows(int64_t n) { return (n + kSmallWindow - 1) / kSmallWindow; }

template <class T>
bool small_usable(int64_t m, int64_t n) {
  return m > 0 && n > 0 && n < kSmallSources && m <= small_pairs<T> / n &&
         m <= kSmallBlocks<T> * 32 * LaneTraits<T>::kLanes;
}

template <class T, int KIND, int NV>
struct SmallFinalize {
  __device__ __forceinline__ static void write(const double (&v)[NV], const Rec<T>* rec,
                                               double* out, double* out2) {
    finalize_values<T, KIND, NV>(v, rec, 0, out, out2, nullptr);
  }
};

template <class Op, class T, int KIND>
struct SmallSweep {
  static constexpr int R = LaneTraits<T>::kLanes;  // one lane of targets per thread
  static constexpr auto kKernel =
      &small_sweep_kernel<Op, T, R, SmallFinalize<T, KIND, Op::NV>>;

  // Resident blocks per SM (asked for when the plan is made: the query also loads the kernel,
  // so that a stream capture after it only launches).
  static int prepare(int* occ) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    const auto key = std::make_pair(reinterpret_cast<const void*>(kKernel), dev);
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_occ.find(key);
    if (it == g_occ.end()) {
      int o = 0;
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, kKernel, kSmallThreads, 0);
      if (e != cudaSuccess) return cuda_fail(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
      it = g_occ.emplace(key, o > 0 ? o : 1).first;
    }
    *occ = it->second;
    return VPM_OK;
  }

  static int launch(SmallArgs a, cudaStream_t st) {
    DevInfo d;
    int occ = 1;
    int rc = device_info(&d);
    if (!rc) rc = prepare(&occ);
    if (rc) return rc;
    // cluster size: the one whose waves of resident blocks walk the fewest windows; a larger
    // cluster costs about a sixteenth of a window more for its reduction
    const double slots = double(d.sms) * (occ < 4 ? occ : 4);
    const int64_t tiles = (int64_t(a.m) + 32 * R - 1) / (32 * R);
    const int64_t windows = small_windows(a.n);
    int S = 1;
    double best = -1.0;
    for (int s = 1; s <= kSmallMaxCluster; s *= 2) {
      const int64_t per = (windows + kSmallWarps * s - 1) / (kSmallWarps * s);
      const double waves = std::ceil(double(tiles * s) / slots);
      const double cost = waves * (double(per) + 0.25) + s / 16.0;
      if (best < 0.0 || cost < best) {
        best = cost;
        S = s;
        a.windows_per_warp = int(per);
      }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(tiles * S));
    cfg.blockDim = dim3(kSmallThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = unsigned(S);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kKernel, a);
    return e == cudaSuccess ? VPM_OK : cuda_fail(e, "small sweep launch");
  }
};

// The one-sided plan of a vector sum; small sums from the caller's arrays take one launch.
template <class Op, class T, int KIND>
int plan_vector(int64_t m, int64_t n, Plan* p, size_t mpb) {
  int rc = Sweep<Op, T>::plan(m, n, p, mpb);
  if (!rc && small_usable<T>(m, n)) {
    int occ = 0;
    rc = SmallSweep<Op, T, KIND>::prepare(&occ);
    p->small = 1;
  }
  return rc;
}

// ---- operator selection -----------------------------------------------------------------
// UC: all cores equal (VPM_UNIFORM_CORE); the probe sums and the kinetic energy keep the
// general form.
template <class T, bool REFINE, bool UC = false>
struct Ops {
  using Vel = OpVel<T, REFINE, UC>;
  using VelAt = OpVelAt<T, REFINE>;
  using VortAt = OpVortAt<T, REFINE>;
  using Stretch = OpStretch<T, REFINE, UC>;
  using Pse = OpPse<T, REFINE, UC>;
  using Ke = OpKe<T, REFINE>;
  using Ens = OpEns<T, REFINE, UC>;
  using VelStretch = OpVelStretch<T, REFINE, UC>;
  using LesStep = OpLesStep<T, REFINE, UC>;
  using VelStretchBoth = OpVelStretchBoth<REFINE, UC>;  // FP32 only
  using VelStretchBothAlt = OpVelStretchBoth<REFINE, UC, VPM_ROT_MINB_ALT>;
  using VelStretchBothSmall = OpVelStretchBoth<REFINE, UC, VPM_ROT_MINB_ALT, 2>;
  using VelStretchBoth64 = OpVelStretchBoth64<UC>;  // FP64 only
  using VelBoth64 = OpVelBoth64<UC>;                // FP64 only
  using PseBoth64 = OpPseBoth64<UC>;                // FP64 only
  using LesStepBoth64 = OpLesStepBoth64<UC>;        // FP64 only
  using StretchBoth64 = OpStretchBoth64<UC>;        // FP64 only
  using RhsVjpBoth64 = OpRhsVjpBoth64<false>;       // FP64 only
  using RhsVjpPseBoth64 = OpRhsVjpBoth64<true>;     // FP64 only
  using VelBoth = OpVelBoth<REFINE, UC>;                // FP32 only
  using PseBoth = OpPseBoth<REFINE, UC>;                // FP32 only
  using LesStepBoth = OpLesStepBoth<REFINE, UC>;        // FP32 only
  using RhsVjpBoth = OpRhsVjpBoth<REFINE, false>;       // FP32 only
  using RhsVjpPseBoth = OpRhsVjpBoth<REFINE, true>;     // FP32 only
  using RhsVjp = OpRhsVjp<T, REFINE, false>;
  using RhsVjpPse = OpRhsVjp<T, REFINE, true>;
  using KeGrad = OpKeGrad<T, REFINE>;
};

bool is_probe(int op) { return op == VPM_OP_INDUCED_VELOCITY_AT || op == VPM_OP_VORTICITY_FIELD_AT; }

template <class T, bool REFINE, bool UC = false>
int plan_op(int op, int64_t m, int64_t n, Plan* p, bool compact,
            size_t max_partial_bytes = kMaxPartialBytes) {
  using O = Ops<T, REFINE, UC>;
  const Budget b(compact, max_partial_bytes, n);
  const size_t mpb = b.one_sided;
  switch (op) {
    case VPM_OP_SELFINDUCED_VELOCITY:
      if constexpr (LaneTraits<T>::kLanes == 2) {
        if (RotSweep<typename O::VelBoth>::usable(m, n, b.both_sides))
          return plan_both32<typename O::VelBoth>(n, p, b);
      } else {
        const int rc = plan_both64<typename O::VelBoth64, true>(m, n, p, b);
        if (rc || p->circle || p->pairs) return rc;
      }
      return plan_vector<typename O::Vel, T, FIN_VEL>(m, n, p, mpb);
    case VPM_OP_TOTAL_HELICITY:
      if constexpr (LaneTraits<T>::kLanes == 1) {
        if (m == n && n > 0) return ScalarSweep<ScalarHel>::plan(n, p);
      }
      return Sweep<typename O::Vel, T>::plan(m, n, p, mpb, true);
    case VPM_OP_INDUCED_VELOCITY_AT:
      return plan_vector<typename O::VelAt, T, FIN_VEL>(m, n, p, mpb);
    case VPM_OP_VORTICITY_FIELD_AT:
      return plan_vector<typename O::VortAt, T, FIN_VORT>(m, n, p, mpb);
    case VPM_OP_STRENGTH_GRADIENTS:
      if constexpr (LaneTraits<T>::kLanes == 1) {
        const int rc = plan_both64<typename O::StretchBoth64, false>(m, n, p, b);
        if (rc || p->circle || p->pairs) return rc;
      }
      return plan_vector<typename O::Stretch, T, FIN_STRETCH>(m, n, p, mpb);
    case VPM_OP_STRENGTH_GRADIENTS_PSE:
      if constexpr (LaneTraits<T>::kLanes == 2) {
        if (RotSweep<typename O::PseBoth>::usable(m, n, b.both_sides))
          return plan_both32<typename O::PseBoth>(n, p, b);
      } else {
        const int rc = plan_both64<typename O::PseBoth64, true>(m, n, p, b);
        if (rc || p->circle || p->pairs) return rc;
      }
      return plan_vector<typename O::Pse, T, FIN_PSE>(m, n, p, mpb);
    case VPM_OP_TOTAL_KINETIC_ENERGY:
      if constexpr (LaneTraits<T>::kLanes == 1) {
        if (m == n && n > 0) return ScalarSweep<ScalarKe>::plan(n, p);
      }
      return Sweep<typename O::Ke, T>::plan(m, n, p, mpb, true);
    case VPM_OP_TOTAL_ENSTROPHY:
      if constexpr (LaneTraits<T>::kLanes == 1) {
        if (m == n && n > 0) return ScalarSweep<ScalarEns>::plan(n, p);
      }
      return Sweep<typename O::Ens, T>::plan(m, n, p, mpb, true);
    case VPM_OP_VELOCITY_AND_STRENGTH_GRADIENTS:
      if constexpr (LaneTraits<T>::kLanes == 2) {
        if (RotSweep<typename O::VelStretchBoth>::usable(m, n, b.both_sides)) {
          // two builds of the fused sum on 768-particle tiles (3 and 2 resident CTAs per SM):
          // take the one whose launches fill the waves better, the 2-CTA build on a tie (it
          // measured equal or faster whenever its waves were as full).  A third on
          // 512-particle tiles (4 targets per lane, 2 CTAs per SM) evaluates pairs at about
          // 0.92 of their rate but makes 2.25x the tile pairs, so it fills the waves where
          // few 768-particle tiles do not (24576: 728 -> 768, 32768: 748 -> 790 Gpairs/s;
          // 49152 and up 6-9 % slower): taken when 0.92 of its fill beats theirs by 1 %.
          constexpr double kSmallTileRate = 0.92;
          Plan pa, pb, pc;
          double ea = 0.0, eb = 0.0, ec = 0.0;
          int rc = RotSweep<typename O::VelStretchBoth>::plan(n, &pa, b.both_sides, &ea);
          if (!rc) rc = RotSweep<typename O::VelStretchBothAlt>::plan(n, &pb, b.both_sides, &eb);
          if (rc) return rc;
          double e = ea;
          if (eb >= ea - 0.01) {
            pb.variant = 1;
            *p = pb;
            e = eb;
          } else {
            *p = pa;
          }
          if (RotSweep<typename O::VelStretchBothSmall>::usable(m, n, b.both_sides)) {
            rc = RotSweep<typename O::VelStretchBothSmall>::plan(n, &pc, b.both_sides, &ec);
            if (rc) return rc;
            if (kSmallTileRate * ec > e + 0.01) {
              pc.variant = 2;
              *p = pc;
            }
          }
          // the one-launch form of the same tiles (the same FP32 sums); of the two builds on
          // 768-particle tiles the one for 2 CTAs per SM
          if (b.compact) return VPM_OK;
          return p->variant == 2
                     ? TriSweep<typename O::VelStretchBothSmall>::plan(n, p, b.both_sides)
                     : TriSweep<typename O::VelStretchBothAlt>::plan(n, p, b.both_sides);
        }
      } else {
        const int rc = plan_both64<typename O::VelStretchBoth64, true>(m, n, p, b);
        if (rc || p->circle || p->pairs) return rc;
      }
      return plan_vector<typename O::VelStretch, T, FIN_VELSTRETCH>(m, n, p, mpb);
    case VPM_OP_LES_STEP_SUMS:
      if constexpr (LaneTraits<T>::kLanes == 2) {
        if (RotSweep<typename O::LesStepBoth>::usable(m, n, b.both_sides))
          return plan_both32<typename O::LesStepBoth>(n, p, b);
      } else {
        const int rc = plan_both64<typename O::LesStepBoth64, true>(m, n, p, b);
        if (rc || p->circle || p->pairs) return rc;
      }
      return Sweep<typename O::LesStep, T>::plan(m, n, p, mpb);
    case VPM_OP_RHS_VJP:
      if constexpr (LaneTraits<T>::kLanes == 2) {
        if (RotSweep<typename O::RhsVjpBoth>::usable(m, n, b.both_sides))
          return plan_both32<typename O::RhsVjpBoth>(n, p, b);
      } else {
        const int rc = plan_both64<typename O::RhsVjpBoth64, false>(m, n, p, b);
        if (rc || p->circle || p->pairs) return rc;
      }
      return Sweep<typename O::RhsVjp, T>::plan(m, n, p, mpb);
    case VPM_OP_RHS_VJP_PSE:
      if constexpr (LaneTraits<T>::kLanes == 2) {
        if (RotSweep<typename O::RhsVjpPseBoth>::usable(m, n, b.both_sides))
          return plan_both32<typename O::RhsVjpPseBoth>(n, p, b);
      } else {
        const int rc = plan_both64<typename O::RhsVjpPseBoth64, false>(m, n, p, b);
        if (rc || p->circle || p->pairs) return rc;
      }
      return Sweep<typename O::RhsVjpPse, T>::plan(m, n, p, mpb);
    case VPM_OP_KINETIC_ENERGY_GRAD:
      return Sweep<typename O::KeGrad, T>::plan(m, n, p, mpb);
    case VPM_OP_LES_TEST_FILTER:
      return Sweep<OpTestFilter<T, REFINE>, T>::plan(m, n, p, mpb);
    default:
      return fail(VPM_ERR_ARG, "unknown op " + std::to_string(op));
  }
}

struct Layout {
  size_t src_off = 0, tgt_off = 0, part_off = 0, total = 0;
  size_t scalar_off = 0;  // LES step sums: one scalar per target, reduced after the finalize
};

template <class T>
size_t op_record_bytes(int op) {
  if (op == VPM_OP_RHS_VJP || op == VPM_OP_RHS_VJP_PSE) return sizeof(RecG<T>);
  if (op == VPM_OP_LES_TEST_FILTER) return sizeof(RecF<T>);
  return sizeof(Rec<T>);
}

template <class T>
Layout layout_for(int op, const Plan& p, int64_t m, int64_t n) {
  Layout L;
  L.src_off = 0;
  size_t off = align_up(size_t(n > 0 ? n : 0) * op_record_bytes<T>(op));
  L.tgt_off = off;
  if (is_probe(op)) off = align_up(off + size_t(m > 0 ? m : 0) * sizeof(Rec<T>));
  L.part_off = off;
  const size_t partials = p.scalar ? ScalarSweep<ScalarKe>::partials(p)
                                   : size_t(p.splits) * p.nv * size_t(m > 0 ? m : 0);
  off = align_up(off + partials * sizeof(double));
  L.scalar_off = off;
  if (op == VPM_OP_LES_STEP_SUMS) off = align_up(off + size_t(m > 0 ? m : 0) * sizeof(double));
  L.total = off;
  return L;
}

template <class T, bool REFINE, bool UC = false>
int workspace_for(int op, int64_t m, int64_t n, Layout* L, Plan* p, bool compact,
                  size_t max_partial_bytes = kMaxPartialBytes) {
  int rc = plan_op<T, REFINE, UC>(op, m, n, p, compact, max_partial_bytes);
  if (rc) return rc;
  *L = layout_for<T>(op, *p, m, n);
  return VPM_OK;
}

struct Call {
  int op;
  const double* tgt;  // probe targets (m,3) or null for self sums
  int64_t m;
  const double* pos;
  const double* str;
  const double* rad;
  const double* nu;
  int64_t n;
  double* out;
  double* out2;
  int ref_extra_4pi;
  void* ws;
  size_t ws_bytes;
  cudaStream_t st;
  const void* records = nullptr;  // pre-packed sources (self sums); null = pack from AoS
  int64_t tgt_begin = 0;          // self sums: targets are records[tgt_begin, tgt_begin + m)
  size_t max_partial_bytes = kMaxPartialBytes;  // caps the source splits of the plan
  bool compact = false;                         // VPM_COMPACT_WORKSPACE
  double* out3 = nullptr;  // VPM_OP_LES_STEP_SUMS: vorticity (m,3)
  double* out4 = nullptr;  // VPM_OP_LES_STEP_SUMS: enstrophy (device scalar)
  const double* aux = nullptr;  // VPM_OP_LES_TEST_FILTER: the filtered fields (n,3)
};

// Whether an output of the call shares memory with one of its inputs.
bool outputs_overlap_inputs(const Call& c) {
  struct Range {
    const double* p;
    int64_t count;
  };
  const Range in[] = {{c.tgt, 3 * c.m}, {c.pos, 3 * c.n}, {c.str, 3 * c.n}, {c.rad, c.n},
                      {c.nu, c.n}};
  for (const double* out : {c.out, c.out2}) {
    if (!out) continue;
    const uintptr_t o = reinterpret_cast<uintptr_t>(out);
    const uintptr_t o_end = o + size_t(3 * c.m) * sizeof(double);
    for (const Range& r : in) {
      if (!r.p) continue;
      const uintptr_t i = reinterpret_cast<uintptr_t>(r.p);
      if (o < i + size_t(r.count) * sizeof(double) && i < o_end) return true;
    }
  }
  return false;
}

template <class T, bool REFINE, bool UC>
int run(const Call& c) {
  using O = Ops<T, REFINE, UC>;
  int rc = check_arch();
  if (rc) return rc;
  const bool scalar = c.op == VPM_OP_TOTAL_KINETIC_ENERGY || c.op == VPM_OP_TOTAL_HELICITY ||
                      c.op == VPM_OP_TOTAL_ENSTROPHY;
  // Empty inputs: zero outputs, no sweep, no workspace needed.
  if (c.m <= 0 || c.n <= 0) {
    if (scalar) {
      write_scalar_kernel<<<1, 1, 0, c.st>>>(c.out, 0.0);
      cudaError_t e = cudaGetLastError();
      return e == cudaSuccess ? VPM_OK : cuda_fail(e, "write launch");
    }
    rc = zero_out(c.out, 3 * (c.m > 0 ? c.m : 0), c.st);
    if (!rc && c.out2) rc = zero_out(c.out2, 3 * (c.m > 0 ? c.m : 0), c.st);
    if (!rc && c.out3) rc = zero_out(c.out3, 3 * (c.m > 0 ? c.m : 0), c.st);
    if (!rc && c.out4) rc = zero_out(c.out4, 1, c.st);
    return rc;
  }

  Plan p;
  Layout L;
  rc = workspace_for<T, REFINE, UC>(c.op, c.m, c.n, &L, &p, c.compact, c.max_partial_bytes);
  if (rc) return rc;
  if (c.ws == nullptr) return fail(VPM_ERR_WORKSPACE, "workspace is null");
  if (reinterpret_cast<uintptr_t>(c.ws) % kAlign != 0)
    return fail(VPM_ERR_ALIGN, "workspace must be 256-byte aligned");
  if (c.ws_bytes < L.total)
    return fail(VPM_ERR_WORKSPACE, "workspace has " + std::to_string(c.ws_bytes) +
                                       " bytes, needs " + std::to_string(L.total));
  // the one launch reads the caller's arrays until its last cluster is done, so outputs that
  // overlap them take the packed route, which copies every input before it writes
  if (p.small && !c.records && !outputs_overlap_inputs(c)) {
    const bool probe = is_probe(c.op);
    const SmallArgs a{probe ? c.tgt : c.pos, probe ? nullptr : c.str, c.nu,     c.pos,
                      c.str,                 c.rad,                   int(c.m), int(c.n),
                      1,                     int(UC),                 c.out,    c.out2};
    switch (c.op) {
      case VPM_OP_SELFINDUCED_VELOCITY:
        return SmallSweep<typename O::Vel, T, FIN_VEL>::launch(a, c.st);
      case VPM_OP_INDUCED_VELOCITY_AT:
        return SmallSweep<typename O::VelAt, T, FIN_VEL>::launch(a, c.st);
      case VPM_OP_VORTICITY_FIELD_AT:
        return SmallSweep<typename O::VortAt, T, FIN_VORT>::launch(a, c.st);
      case VPM_OP_STRENGTH_GRADIENTS:
        return SmallSweep<typename O::Stretch, T, FIN_STRETCH>::launch(a, c.st);
      case VPM_OP_STRENGTH_GRADIENTS_PSE:
        return SmallSweep<typename O::Pse, T, FIN_PSE>::launch(a, c.st);
      case VPM_OP_VELOCITY_AND_STRENGTH_GRADIENTS:
        return SmallSweep<typename O::VelStretch, T, FIN_VELSTRETCH>::launch(a, c.st);
      default:
        break;
    }
  }
  char* ws = static_cast<char*>(c.ws);
  Rec<T>* src = c.records ? const_cast<Rec<T>*>(static_cast<const Rec<T>*>(c.records))
                          : reinterpret_cast<Rec<T>*>(ws + L.src_off);
  Rec<T>* tgt = is_probe(c.op) ? reinterpret_cast<Rec<T>*>(ws + L.tgt_off) : src + c.tgt_begin;
  double* part = reinterpret_cast<double*>(ws + L.part_off);

  if (!c.records) {
    rc = pack<T>(c.pos, c.str, c.rad, c.nu, c.n, src, c.st, UC);
    if (rc) return rc;
  }
  if (is_probe(c.op)) {
    rc = pack<T>(c.tgt, nullptr, nullptr, nullptr, c.m, tgt, c.st);
    if (rc) return rc;
  }

  switch (c.op) {
    case VPM_OP_SELFINDUCED_VELOCITY:
      rc = VPM_OK;
      if constexpr (LaneTraits<T>::kLanes == 1) {
        if (p.circle)
          return CircleSweep<typename O::VelBoth64>::launch(
              p, src, c.n, part, SetsFinalize<double, FIN_VEL, 3>{src, c.out, nullptr, nullptr, nullptr},
              c.st);
        if (p.triangle)
          return TriSweep<typename O::VelBoth64>::launch(
              p, src, c.n, part, SetsFinalize<double, FIN_VEL, 3>{src, c.out, nullptr, nullptr, nullptr},
              c.st);
      } else if (p.triangle) {
        return TriSweep<typename O::VelBoth>::launch(
            p, src, c.n, part, SetsFinalize<T, FIN_VEL, 3>{src, c.out, nullptr, nullptr, nullptr},
            c.st);
      }
      if (p.pairs) {  // m == n: the targets are all the records (tgt_begin == 0)
        if constexpr (LaneTraits<T>::kLanes == 2)
          rc = RotSweep<typename O::VelBoth>::launch(p, src, c.n, part, c.st);
        else
          rc = RotSweep<typename O::VelBoth64>::launch(p, src, c.n, part, c.st);
      }
      if (!p.pairs)
        rc = Sweep<typename O::Vel, T>::launch(p, tgt, c.m, c.tgt_begin, src, c.n, part, c.st);
      if (!rc) rc = finalize_vec<T, FIN_VEL, 3>(part, p.splits, c.m, tgt, c.out, nullptr, c.st);
      return rc;
    case VPM_OP_INDUCED_VELOCITY_AT:
      rc = Sweep<typename O::VelAt, T>::launch(p, tgt, c.m, c.tgt_begin, src, c.n, part, c.st);
      if (!rc) rc = finalize_vec<T, FIN_VEL, 3>(part, p.splits, c.m, tgt, c.out, nullptr, c.st);
      return rc;
    case VPM_OP_VORTICITY_FIELD_AT:
      rc = Sweep<typename O::VortAt, T>::launch(p, tgt, c.m, c.tgt_begin, src, c.n, part, c.st);
      if (!rc) rc = finalize_vec<T, FIN_VORT, 3>(part, p.splits, c.m, tgt, c.out, nullptr, c.st);
      return rc;
    case VPM_OP_STRENGTH_GRADIENTS:
      if constexpr (LaneTraits<T>::kLanes == 1) {
        if (p.circle)
          return CircleSweep<typename O::StretchBoth64>::launch(
              p, src, c.n, part,
              SetsFinalize<double, FIN_STRETCH, 6>{src, c.out, nullptr, nullptr, nullptr}, c.st);
        if (p.pairs) rc = RotSweep<typename O::StretchBoth64>::launch(p, src, c.n, part, c.st);
      }
      if (!p.pairs)
        rc = Sweep<typename O::Stretch, T>::launch(p, tgt, c.m, c.tgt_begin, src, c.n, part,
                                                   c.st);
      if (!rc)
        rc = finalize_vec<T, FIN_STRETCH, 6>(part, p.splits, c.m, tgt, c.out, nullptr, c.st);
      return rc;
    case VPM_OP_STRENGTH_GRADIENTS_PSE:
      rc = VPM_OK;
      if constexpr (LaneTraits<T>::kLanes == 1) {
        if (p.circle)
          return CircleSweep<typename O::PseBoth64>::launch(
              p, src, c.n, part, SetsFinalize<double, FIN_PSE, 3>{src, c.out, nullptr, nullptr, nullptr},
              c.st);
        if (p.triangle)
          return TriSweep<typename O::PseBoth64>::launch(
              p, src, c.n, part, SetsFinalize<double, FIN_PSE, 3>{src, c.out, nullptr, nullptr, nullptr},
              c.st);
      } else if (p.triangle) {
        return TriSweep<typename O::PseBoth>::launch(
            p, src, c.n, part, SetsFinalize<T, FIN_PSE, 3>{src, c.out, nullptr, nullptr, nullptr},
            c.st);
      }
      if (p.pairs) {
        if constexpr (LaneTraits<T>::kLanes == 2)
          rc = RotSweep<typename O::PseBoth>::launch(p, src, c.n, part, c.st);
        else
          rc = RotSweep<typename O::PseBoth64>::launch(p, src, c.n, part, c.st);
      }
      if (!p.pairs)
        rc = Sweep<typename O::Pse, T>::launch(p, tgt, c.m, c.tgt_begin, src, c.n, part, c.st);
      if (!rc) rc = finalize_vec<T, FIN_PSE, 3>(part, p.splits, c.m, tgt, c.out, nullptr, c.st);
      return rc;
    case VPM_OP_VELOCITY_AND_STRENGTH_GRADIENTS:
      if constexpr (LaneTraits<T>::kLanes == 2) {
        if (p.triangle) {
          const SetsFinalize<T, FIN_VELSTRETCH, 9> fin{src, c.out, c.out2, nullptr, nullptr};
          if (p.variant == 2)
            return TriSweep<typename O::VelStretchBothSmall>::launch(p, src, c.n, part, fin, c.st);
          return TriSweep<typename O::VelStretchBothAlt>::launch(p, src, c.n, part, fin, c.st);
        }
        if (p.pairs && p.variant == 2)  // m == n: the targets are all the records
          rc = RotSweep<typename O::VelStretchBothSmall>::launch(p, src, c.n, part, c.st);
        else if (p.pairs && p.variant == 1)
          rc = RotSweep<typename O::VelStretchBothAlt>::launch(p, src, c.n, part, c.st);
        else if (p.pairs)
          rc = RotSweep<typename O::VelStretchBoth>::launch(p, src, c.n, part, c.st);
        else
          rc = Sweep<typename O::VelStretch, T>::launch(p, tgt, c.m, c.tgt_begin, src, c.n,
                                                        part, c.st);
      } else if (p.circle) {
        return CircleSweep<typename O::VelStretchBoth64>::launch(
            p, src, c.n, part,
            SetsFinalize<double, FIN_VELSTRETCH, 9>{src, c.out, c.out2, nullptr, nullptr}, c.st);
      } else if (p.triangle) {
        return TriSweep<typename O::VelStretchBoth64>::launch(
            p, src, c.n, part,
            SetsFinalize<double, FIN_VELSTRETCH, 9>{src, c.out, c.out2, nullptr, nullptr}, c.st);
      } else if (p.pairs) {
        rc = RotSweep<typename O::VelStretchBoth64>::launch(p, src, c.n, part, c.st);
      } else {
        rc = Sweep<typename O::VelStretch, T>::launch(p, tgt, c.m, c.tgt_begin, src, c.n, part,
                                                      c.st);
      }
      if (!rc)
        rc = finalize_vec<T, FIN_VELSTRETCH, O::VelStretch::NV>(part, p.splits, c.m, tgt, c.out,
                                                               c.out2, c.st);
      return rc;
    case VPM_OP_LES_STEP_SUMS: {
      using Op = typename O::LesStep;
      rc = VPM_OK;
      if (p.pairs && !p.triangle) {
        if constexpr (LaneTraits<T>::kLanes == 2)
          rc = RotSweep<typename O::LesStepBoth>::launch(p, src, c.n, part, c.st);
        else
          rc = RotSweep<typename O::LesStepBoth64>::launch(p, src, c.n, part, c.st);
        if (rc) return rc;
      }
      double scale = 1.0 / (8.0 * kPi);
      if (c.ref_extra_4pi) scale /= 4.0 * kPi;
      // every target's scalar a_i . E_i: from the both-sides sums sum_j ke (a_i . a_j) (value
      // 12), taken once per unordered pair, so doubled
      double* scalar = reinterpret_cast<double*>(ws + L.scalar_off);
      constexpr int NVB = O::LesStepBoth::NV;
      static_assert(O::LesStepBoth64::NV == NVB, "one row layout for both precisions");
      bool done = false;
      if constexpr (LaneTraits<T>::kLanes == 1) {
        if (p.circle) {
          rc = CircleSweep<typename O::LesStepBoth64>::launch(
              p, src, c.n, part,
              SetsFinalize<double, FIN_LES, NVB>{src, c.out, c.out2, c.out3, scalar}, c.st);
          scale *= 2.0;
          done = true;
        }
        if (p.triangle) {
          rc = TriSweep<typename O::LesStepBoth64>::launch(
              p, src, c.n, part,
              SetsFinalize<double, FIN_LES, NVB>{src, c.out, c.out2, c.out3, scalar}, c.st);
          scale *= 2.0;
          done = true;
        }
      } else if (p.triangle) {
        rc = TriSweep<typename O::LesStepBoth>::launch(
            p, src, c.n, part,
            SetsFinalize<T, FIN_LES, NVB>{src, c.out, c.out2, c.out3, scalar}, c.st);
        scale *= 2.0;
        done = true;
      }
      if (!done && p.pairs) {
        rc = finalize_vec<T, FIN_LES, NVB>(part, p.splits, c.m, tgt, c.out, c.out2, c.st, c.out3,
                                           scalar);
        scale *= 2.0;
      } else if (!done) {
        rc = Sweep<Op, T>::launch(p, tgt, c.m, c.tgt_begin, src, c.n, part, c.st);
        if (!rc)
          rc = finalize_vec<T, FIN_LES, Op::NV>(part, p.splits, c.m, tgt, c.out, c.out2, c.st,
                                                c.out3, scalar);
      }
      if (rc) return rc;
      finalize_sum_kernel<<<1, kReduceThreads, 0, c.st>>>(scalar, c.m, scale, c.out4);
      cudaError_t e = cudaGetLastError();
      return e == cudaSuccess ? VPM_OK : cuda_fail(e, "reduce launch");
    }
    case VPM_OP_TOTAL_KINETIC_ENERGY:
    case VPM_OP_TOTAL_HELICITY:
    case VPM_OP_TOTAL_ENSTROPHY: {
      double scale = 0.0;
      if constexpr (LaneTraits<T>::kLanes == 1) {
        if (p.scalar) {
          const double extra = c.ref_extra_4pi ? 4.0 * kPi : 1.0;
          if (c.op == VPM_OP_TOTAL_KINETIC_ENERGY)
            return ScalarSweep<ScalarKe>::launch(p, src, c.n, part, 1.0 / (16.0 * kPi), c.out,
                                                 c.st);
          if (c.op == VPM_OP_TOTAL_HELICITY)
            return ScalarSweep<ScalarHel>::launch(p, src, c.n, part, -1.0 / (4.0 * kPi) / extra,
                                                  c.out, c.st);
          return ScalarSweep<ScalarEns>::launch(p, src, c.n, part, 1.0 / (8.0 * kPi) / extra,
                                                c.out, c.st);
        }
      }
      if (c.op == VPM_OP_TOTAL_KINETIC_ENERGY) {
        rc = Sweep<typename O::Ke, T>::launch(p, tgt, c.m, c.tgt_begin, src, c.n, part, c.st);
        scale = 1.0 / (16.0 * kPi);
      } else if (c.op == VPM_OP_TOTAL_HELICITY) {
        rc = Sweep<typename O::Vel, T>::launch(p, tgt, c.m, c.tgt_begin, src, c.n, part, c.st);
        scale = -1.0 / (4.0 * kPi);
        if (c.ref_extra_4pi) scale /= 4.0 * kPi;
      } else {
        rc = Sweep<typename O::Ens, T>::launch(p, tgt, c.m, c.tgt_begin, src, c.n, part, c.st);
        scale = 1.0 / (8.0 * kPi);
        if (c.ref_extra_4pi) scale /= 4.0 * kPi;
      }
      if (rc) return rc;
      finalize_dot_kernel<T><<<1, kReduceThreads, 0, c.st>>>(part, p.splits, c.m, tgt, scale,
                                                             c.out);
      cudaError_t e = cudaGetLastError();
      return e == cudaSuccess ? VPM_OK : cuda_fail(e, "reduce launch");
    }
    default:
      return fail(VPM_ERR_ARG, "unknown op " + std::to_string(c.op));
  }
}

// ---- LES test filter (least-squares dynamic coefficient) ----------------------------------
template <class E>
__global__ void pack_filter_kernel(const double* __restrict__ pos, const double* __restrict__ str,
                                   const double* __restrict__ rad, const double* __restrict__ f,
                                   int64_t n, RecF<E>* __restrict__ out) {
  const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  RecF<E> r;
  set_elem(r.x, pos[3 * i]);
  set_elem(r.y, pos[3 * i + 1]);
  set_elem(r.z, pos[3 * i + 2]);
  set_elem(r.s, rad[i]);
  set_elem(r.ax, str[3 * i]);
  set_elem(r.ay, str[3 * i + 1]);
  set_elem(r.az, str[3 * i + 2]);
  set_elem(r.f1, f[3 * i]);
  set_elem(r.f2, f[3 * i + 1]);
  set_elem(r.pad, 0.0);
  out[i] = r;
}

// w_hat (m,3) and the two filtered fields (m,3; third column 0), both with the zeta kernel's
// 7.5/(4 pi) as in vpm_vorticity_field_at.
struct SetsFinalizeFilter {
  double *w_hat, *f_hat;
  __device__ __forceinline__ void write(const double (&v)[5], int64_t i) const {
    const double c = 7.5 * kOneOver4Pi;
    w_hat[3 * i] = v[0] * c;
    w_hat[3 * i + 1] = v[1] * c;
    w_hat[3 * i + 2] = v[2] * c;
    f_hat[3 * i] = v[3] * c;
    f_hat[3 * i + 1] = v[4] * c;
    f_hat[3 * i + 2] = 0.0;
  }
};

template <class T, bool REFINE>
int run_filter(const Call& c) {
  using Op = OpTestFilter<T, REFINE>;
  int rc = check_arch();
  if (rc) return rc;
  if (c.n == 0) return VPM_OK;
  Plan p;
  Layout L;
  rc = workspace_for<T, REFINE>(c.op, c.n, c.n, &L, &p, c.compact, c.max_partial_bytes);
  if (rc) return rc;
  if (c.ws == nullptr) return fail(VPM_ERR_WORKSPACE, "workspace is null");
  if (reinterpret_cast<uintptr_t>(c.ws) % kAlign != 0)
    return fail(VPM_ERR_ALIGN, "workspace must be 256-byte aligned");
  if (c.ws_bytes < L.total)
    return fail(VPM_ERR_WORKSPACE, "workspace has " + std::to_string(c.ws_bytes) +
                                       " bytes, needs " + std::to_string(L.total));
  char* ws = static_cast<char*>(c.ws);
  RecF<T>* rec = reinterpret_cast<RecF<T>*>(ws + L.src_off);
  double* part = reinterpret_cast<double*>(ws + L.part_off);
  const unsigned blocks = unsigned((c.n + 255) / 256);
  pack_filter_kernel<T><<<blocks, 256, 0, c.st>>>(c.pos, c.str, c.rad, c.aux, c.n, rec);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "pack launch");
  rc = Sweep<Op, T>::launch(p, rec, c.n, 0, rec, c.n, part, c.st);
  if (rc) return rc;
  return finalize<5>(part, p.splits, c.n, SetsFinalizeFilter{c.out, c.out2}, c.st);
}

// Flags of a precision code.
constexpr int kPrecisionFlags = VPM_UNIFORM_CORE | VPM_COMPACT_WORKSPACE;

// Decoded precision code: compute type, Newton-refined rsqrt, uniform cores.
template <class T, bool REFINE, bool UC>
struct Prec {
  using type = T;
  static constexpr bool refine = REFINE, uc = UC;
};

template <class F>
int with_precision(int precision, F&& f) {
  const bool uc = (precision & VPM_UNIFORM_CORE) != 0;
  switch (precision & ~kPrecisionFlags) {
    case VPM_FP64:
      return uc ? f(Prec<double, false, true>{}) : f(Prec<double, false, false>{});
    case VPM_FP32C:
      return uc ? f(Prec<float2, false, true>{}) : f(Prec<float2, false, false>{});
    case VPM_FP32C_REFINED:
      return uc ? f(Prec<float2, true, true>{}) : f(Prec<float2, true, false>{});
    default:
      return fail(VPM_ERR_ARG, "unknown precision " + std::to_string(precision));
  }
}

int dispatch(Call c, int precision) {
  c.compact = (precision & VPM_COMPACT_WORKSPACE) != 0;
  if (c.n < 0 || c.m < 0) return fail(VPM_ERR_ARG, "negative size");
  if (c.records) {
    if (is_probe(c.op)) return fail(VPM_ERR_ARG, "record entry points are for self sums");
    if (c.tgt_begin < 0 || c.tgt_begin + c.m > c.n)
      return fail(VPM_ERR_ARG, "target range outside the records");
    if (reinterpret_cast<uintptr_t>(c.records) % 16 != 0)
      return fail(VPM_ERR_ALIGN, "records must be 16-byte aligned");
  } else {
    if (c.n > 0 && (!c.pos || !c.rad)) return fail(VPM_ERR_ARG, "null input pointer");
    if (c.n > 0 && !c.str) return fail(VPM_ERR_ARG, "null strengths pointer");
  }
  if (c.m > 0 && !c.out) return fail(VPM_ERR_ARG, "null output pointer");
  if (is_probe(c.op) && c.m > 0 && !c.tgt) return fail(VPM_ERR_ARG, "null targets pointer");
  if (c.op == VPM_OP_STRENGTH_GRADIENTS_PSE && c.n > 0 && !c.nu && !c.records)
    return fail(VPM_ERR_ARG, "null viscosities pointer");
  if ((c.op == VPM_OP_VELOCITY_AND_STRENGTH_GRADIENTS || c.op == VPM_OP_LES_STEP_SUMS) &&
      c.m > 0 && !c.out2)
    return fail(VPM_ERR_ARG, "null second output pointer");
  if (c.op == VPM_OP_LES_STEP_SUMS && ((c.m > 0 && !c.out3) || !c.out4))
    return fail(VPM_ERR_ARG, "null vorticity or enstrophy pointer");
  return with_precision(precision, [&](auto P) {
    using Pp = decltype(P);
    return run<typename Pp::type, Pp::refine, Pp::uc>(c);
  });
}

struct GradCall {
  int op;
  const double *pos, *str, *rad, *nu, *gu, *gs;
  int64_t n;
  double *ox, *oa, *os, *onu;
  void* ws;
  size_t ws_bytes;
  cudaStream_t st;
  bool compact = false;  // VPM_COMPACT_WORKSPACE
};

template <class T, bool REFINE>
int run_grad(const GradCall& c) {
  using O = Ops<T, REFINE>;
  int rc = check_arch();
  if (rc) return rc;
  if (c.n == 0) return VPM_OK;
  Plan p;
  Layout L;
  rc = workspace_for<T, REFINE>(c.op, c.n, c.n, &L, &p, c.compact);
  if (rc) return rc;
  if (c.ws == nullptr) return fail(VPM_ERR_WORKSPACE, "workspace is null");
  if (reinterpret_cast<uintptr_t>(c.ws) % kAlign != 0)
    return fail(VPM_ERR_ALIGN, "workspace must be 256-byte aligned");
  if (c.ws_bytes < L.total)
    return fail(VPM_ERR_WORKSPACE, "workspace has " + std::to_string(c.ws_bytes) +
                                       " bytes, needs " + std::to_string(L.total));
  char* ws = static_cast<char*>(c.ws);
  double* part = reinterpret_cast<double*>(ws + L.part_off);
  const unsigned blocks = unsigned((c.n + 255) / 256);
  cudaError_t e;
  if (c.op == VPM_OP_KINETIC_ENERGY_GRAD) {
    Rec<T>* rec = reinterpret_cast<Rec<T>*>(ws + L.src_off);
    rc = pack<T>(c.pos, c.str, c.rad, nullptr, c.n, rec, c.st);
    if (!rc) rc = Sweep<typename O::KeGrad, T>::launch(p, rec, c.n, 0, rec, c.n, part, c.st);
    if (rc) return rc;
    return finalize<7>(part, p.splits, c.n, SetsFinalizeKeGrad{c.ox, c.oa, c.os}, c.st);
  }
  RecG<T>* rec = reinterpret_cast<RecG<T>*>(ws + L.src_off);
  pack_grad_kernel<T><<<blocks, 256, 0, c.st>>>(c.pos, c.str, c.rad, c.nu, c.gu, c.gs, c.n, rec);
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "pack launch");
  if (c.op == VPM_OP_RHS_VJP_PSE) {
    rc = VPM_OK;
    if constexpr (LaneTraits<T>::kLanes == 2) {
      if (p.triangle)
        return TriSweep<typename O::RhsVjpPseBoth>::launch(
            p, rec, c.n, part, SetsFinalizeVjp<T, true>{rec, c.ox, c.oa, c.os, c.onu}, c.st);
      if (p.pairs) rc = RotSweep<typename O::RhsVjpPseBoth>::launch(p, rec, c.n, part, c.st);
    } else {
      if (p.circle)
        return CircleSweep<typename O::RhsVjpPseBoth64>::launch(
            p, rec, c.n, part, SetsFinalizeVjp<double, true>{rec, c.ox, c.oa, c.os, c.onu}, c.st);
      if (p.pairs) rc = RotSweep<typename O::RhsVjpPseBoth64>::launch(p, rec, c.n, part, c.st);
    }
    if (!p.pairs)
      rc = Sweep<typename O::RhsVjpPse, T>::launch(p, rec, c.n, 0, rec, c.n, part, c.st);
    if (rc) return rc;
    rc = finalize<O::RhsVjpPse::NV>(part, p.splits, c.n,
                             SetsFinalizeVjp<T, true>{rec, c.ox, c.oa, c.os, c.onu}, c.st);
  } else {
    rc = VPM_OK;
    if constexpr (LaneTraits<T>::kLanes == 2) {
      if (p.triangle)
        return TriSweep<typename O::RhsVjpBoth>::launch(
            p, rec, c.n, part, SetsFinalizeVjp<T, false>{rec, c.ox, c.oa, c.os, c.onu}, c.st);
      if (p.pairs) rc = RotSweep<typename O::RhsVjpBoth>::launch(p, rec, c.n, part, c.st);
    } else {
      if (p.circle)
        return CircleSweep<typename O::RhsVjpBoth64>::launch(
            p, rec, c.n, part, SetsFinalizeVjp<double, false>{rec, c.ox, c.oa, c.os, c.onu}, c.st);
      if (p.pairs) rc = RotSweep<typename O::RhsVjpBoth64>::launch(p, rec, c.n, part, c.st);
    }
    if (!p.pairs) rc = Sweep<typename O::RhsVjp, T>::launch(p, rec, c.n, 0, rec, c.n, part, c.st);
    if (rc) return rc;
    rc = finalize<O::RhsVjp::NV>(part, p.splits, c.n,
                             SetsFinalizeVjp<T, false>{rec, c.ox, c.oa, c.os, c.onu}, c.st);
  }
  return rc;
}

int dispatch_grad(GradCall c, int precision) {
  c.compact = (precision & VPM_COMPACT_WORKSPACE) != 0;
  precision &= ~kPrecisionFlags;  // the adjoint keeps the general pair core
  if (c.n < 0) return fail(VPM_ERR_ARG, "negative size");
  if (c.n > 0 && (!c.pos || !c.str || !c.rad || !c.ox || !c.oa || !c.os))
    return fail(VPM_ERR_ARG, "null pointer");
  if (c.op != VPM_OP_KINETIC_ENERGY_GRAD && c.n > 0 && (!c.gu || !c.gs))
    return fail(VPM_ERR_ARG, "null cotangent pointer");
  switch (precision) {
    case VPM_FP64:
      return run_grad<double, false>(c);
    case VPM_FP32C:
      return run_grad<float2, false>(c);
    case VPM_FP32C_REFINED:
      return run_grad<float2, true>(c);
    default:
      return fail(VPM_ERR_ARG, "unknown precision " + std::to_string(precision));
  }
}


// ---- scratch for the no-allocation entry point --------------------------------------------
// Some callers may not allocate device memory at all: a solver plugin that runs inside a
// host application which owns the whole GPU memory budget through its own pool, or a
// fixed-latency loop where a cudaMalloc (which may synchronise the device, and fails once
// memory is exhausted) is not permitted.  For them one entry point takes its scratch from
// this array, which the library image reserves on every GPU that loads it, until exit.
// Host code must not use the array's name as a device address: the address is fetched per
// device with cudaGetSymbolAddress.
constexpr int64_t kNoAllocMaxN = VPM_NOALLOC_MAX_N;
constexpr size_t kNoAllocScratchBytes = VPM_NOALLOC_SCRATCH_BYTES;
constexpr size_t kNoAllocRecordBytes = size_t(kNoAllocMaxN) * 64;  // packed records
static_assert(kNoAllocRecordBytes % kAlign == 0, "record region stays 256-byte aligned");
static_assert(kNoAllocScratchBytes > kNoAllocRecordBytes, "room for partials");

// (device, driver context) -> device address of the scratch in that context.  A __device__
// array has one address per context, so a host application that makes another context
// current on the same device gets its own lookup.
std::map<std::pair<int, void*>, void*> g_noalloc_addr;

int noalloc_scratch(void** out);

// ---- bounded-wait self-test -----------------------------------------------------------------
// One block waits on an mbarrier phase that nothing completes (16 transaction bytes are
// expected and never sent).  mbar_wait_bounded gives up after its time limit, records
// VPM_DEVERR_WAIT_TIMEOUT and the kernel returns: the same path a sweep takes when a tile copy
// never lands.  No copy is issued, so nothing is in flight when the block exits.
__global__ void bounded_wait_selftest_kernel(int* __restrict__ result) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
  }
  __syncthreads();
  if (threadIdx.x == 0) mbar_arrive_expect_tx(&bar, 16);
  __syncthreads();
  const bool ok = mbar_wait_bounded(&bar, 0);
  if (__syncthreads_or(!ok) && threadIdx.x == 0) result[0] = 1;
}

// ---- FMA throughput kernels ------------------------------------------------------------
template <class T>
__global__ void fma_peak_kernel(int iters, T* sink) {
  T a[16];
  const T m = T(1.0) - T(1e-7) * T(threadIdx.x & 7);
  const T b = T(1e-9) * T(blockIdx.x & 3);
#pragma unroll
  for (int k = 0; k < 16; ++k) a[k] = T(threadIdx.x + k);
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int k = 0; k < 16; ++k) a[k] = fma(a[k], m, b);
  }
  T s = 0;
#pragma unroll
  for (int k = 0; k < 16; ++k) s += a[k];
  sink[int64_t(blockIdx.x) * blockDim.x + threadIdx.x] = s;
}

// Packed FP32 FMA throughput: 16 independent chains of FFMA2 (two FP32 lanes each).
__global__ void ffma2_peak_kernel(int iters, float* sink) {
  float2 a[16];
  const float2 m = make_float2(1.0f - 1e-7f * float(threadIdx.x & 7), 1.0f - 2e-7f);
  const float2 b = make_float2(1e-9f * float(blockIdx.x & 3), 1e-9f);
#pragma unroll
  for (int k = 0; k < 16; ++k) a[k] = make_float2(float(threadIdx.x + k), float(k));
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int k = 0; k < 16; ++k) a[k] = fma(a[k], m, b);
  }
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < 16; ++k) s += a[k].x + a[k].y;
  sink[int64_t(blockIdx.x) * blockDim.x + threadIdx.x] = s;
}

// Mixed FP32 FMA throughput: 8 packed FFMA2 chains and 16 scalar FFMA chains per thread (32
// lane FMAs per iteration in 24 instructions).
__global__ void ffma_mixed_peak_kernel(int iters, float* sink) {
  float2 a[8];
  float c[16];
  const float2 m = make_float2(1.0f - 1e-7f * float(threadIdx.x & 7), 1.0f - 2e-7f);
  const float2 b = make_float2(1e-9f * float(blockIdx.x & 3), 1e-9f);
#pragma unroll
  for (int k = 0; k < 8; ++k) a[k] = make_float2(float(threadIdx.x + k), float(k));
#pragma unroll
  for (int k = 0; k < 16; ++k) c[k] = float(threadIdx.x + 2 * k);
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      a[k] = fma(a[k], m, b);
      c[2 * k] = fmaf(c[2 * k], m.x, b.x);
      c[2 * k + 1] = fmaf(c[2 * k + 1], m.y, b.y);
    }
  }
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < 8; ++k) s += a[k].x + a[k].y + c[2 * k] + c[2 * k + 1];
  sink[int64_t(blockIdx.x) * blockDim.x + threadIdx.x] = s;
}

// MUFU (SFU) throughput: 16 independent chains of rsqrt.approx per thread; the one FADD per
// step runs on the FMA pipe, which has 8x the lanes of the SFU, so the SFU bounds the loop.
__global__ void rsqrt_peak_kernel(int iters, float* sink) {
  float a[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) a[k] = 1.0f + 1e-3f * float(threadIdx.x) + float(k);
  for (int it = 0; it < iters; ++it) {
#pragma unroll
    for (int k = 0; k < 16; ++k) a[k] = rsqrt_approx(a[k] + 0.5f);
  }
  float s = 0.f;
#pragma unroll
  for (int k = 0; k < 16; ++k) s += a[k];
  sink[int64_t(blockIdx.x) * blockDim.x + threadIdx.x] = s;
}

}  // namespace

// File-scope scratch of vpm_selfinduced_velocity_noalloc (see noalloc_scratch).
static __device__ __align__(256) unsigned char g_noalloc_scratch[VPM_NOALLOC_SCRATCH_BYTES];

namespace {
// The driver context current on the calling thread (cuCtxGetCurrent, reached through the
// runtime's driver entry-point table so the library needs no link against libcuda).
int current_context(void** ctx) {
  using CtxGetCurrent = CUresult (*)(CUcontext*);
  static CtxGetCurrent fn = nullptr;
  static std::once_flag once;
  static cudaError_t lookup = cudaSuccess;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    lookup = cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q);
    if (lookup == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<CtxGetCurrent>(p);
  });
  if (lookup != cudaSuccess) return cuda_fail(lookup, "cudaGetDriverEntryPoint(cuCtxGetCurrent)");
  if (!fn) return fail(VPM_ERR_CUDA, "cuCtxGetCurrent not found in the driver");
  CUcontext c = nullptr;
  if (fn(&c) != CUDA_SUCCESS || !c) return fail(VPM_ERR_CUDA, "no current CUDA context");
  *ctx = c;
  return VPM_OK;
}

// Device address of g_noalloc_scratch in the current context, looked up once per (device,
// context) with that context current, and cached.
int noalloc_scratch(void** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  void* ctx = nullptr;
  int rc = current_context(&ctx);
  if (rc) return rc;
  std::lock_guard<std::mutex> lk(g_mu);
  const auto key = std::make_pair(dev, ctx);
  auto it = g_noalloc_addr.find(key);
  if (it == g_noalloc_addr.end()) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(no-allocation scratch)");
    it = g_noalloc_addr.emplace(key, p).first;
  }
  *out = it->second;
  return VPM_OK;
}
}  // namespace
}  // namespace vpm

using namespace vpm;

// ---- pair shards across GPUs: the fused sum's both-sides schedule split by tile ranges ----
// Calls f(RotSweep<X>{}, plan) for the both-sides build the planner takes for a self sum of n
// particles (every rank plans the same n, so all ranks use the same tiles and launch sizes).
template <class T, bool REFINE, bool UC, class F>
int with_fused_both(int64_t n, F&& f) {
  using O = Ops<T, REFINE, UC>;
  Plan p;
  int rc = plan_op<T, REFINE, UC>(VPM_OP_VELOCITY_AND_STRENGTH_GRADIENTS, n, n, &p, false);
  if (rc) return rc;
  if (!p.pairs)
    return fail(VPM_ERR_ARG, "n = " + std::to_string(n) +
                                 " does not take the both-sides schedule "
                                 "(vpm_set_symmetric_min_n); shard the targets instead");
  if constexpr (LaneTraits<T>::kLanes != 2) {
    return f(RotSweep<typename O::VelStretchBoth64>{}, p);
  } else {
    if (p.variant == 2) return f(RotSweep<typename O::VelStretchBothSmall>{}, p);
    if (p.variant == 1) return f(RotSweep<typename O::VelStretchBothAlt>{}, p);
    return f(RotSweep<typename O::VelStretchBoth>{}, p);
  }
}

extern "C" {

int vpm_abi_version(void) { return VPM_ABI_VERSION; }

const char* vpm_last_error(void) { return g_last_error.c_str(); }

int vpm_check_device(void) { return check_arch(); }

int vpm_binary_info(int* binary_version, int* ptx_version) {
  if (!binary_version || !ptx_version) return fail(VPM_ERR_ARG, "null result pointer");
  cudaFuncAttributes fa;
  cudaError_t e = cudaFuncGetAttributes(&fa, reinterpret_cast<const void*>(&zero_kernel));
  if (e != cudaSuccess) return cuda_fail(e, "cudaFuncGetAttributes");
  *binary_version = fa.binaryVersion;
  *ptx_version = fa.ptxVersion;
  return VPM_OK;
}

int vpm_device_errors(int* out, int clear) {
  int v = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&v, g_device_errors, sizeof(int));
  if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyFromSymbol");
  if (out) *out = v;
  if (clear) {
    const int z = 0;
    e = cudaMemcpyToSymbol(g_device_errors, &z, sizeof(int));
    if (e != cudaSuccess) return cuda_fail(e, "cudaMemcpyToSymbol");
  }
  return VPM_OK;
}

size_t vpm_workspace_bytes(int op, int precision, int64_t m, int64_t n) {
  if (op == VPM_OP_RHS_VJP || op == VPM_OP_RHS_VJP_PSE || op == VPM_OP_KINETIC_ENERGY_GRAD)
    precision &= ~VPM_UNIFORM_CORE;
  size_t total = 0;
  const int rc = with_precision(precision, [&](auto P) {
    using Pp = decltype(P);
    Plan p;
    Layout L;
    const int r = workspace_for<typename Pp::type, Pp::refine, Pp::uc>(
        op, m, n, &L, &p, (precision & VPM_COMPACT_WORKSPACE) != 0);
    if (!r) total = L.total;
    return r;
  });
  return rc ? 0 : total;
}

int vpm_pairs_layout(int op, int precision, int64_t n, int64_t* tiles, int64_t* pairs,
                     int* pairs_per_launch, int* values, size_t* workspace_bytes) {
  if (op != VPM_OP_VELOCITY_AND_STRENGTH_GRADIENTS)
    return fail(VPM_ERR_ARG, "pair shards are built for the fused velocity + stretching sum");
  if (n < 0) return fail(VPM_ERR_ARG, "negative size");
  return with_precision(precision, [&](auto P) {
    using Pp = decltype(P);
    return with_fused_both<typename Pp::type, Pp::refine, Pp::uc>(n, [&](auto rs,
                                                                        const Plan& p) {
      using RS = decltype(rs);
      const int64_t nt = RS::tiles(n);
      if (tiles) *tiles = nt;
      if (pairs) *pairs = nt / 2;
      if (pairs_per_launch) *pairs_per_launch = p.pairs;
      if (values) *values = RS::NV;
      if (workspace_bytes) *workspace_bytes = size_t(RS::sets(p.pairs)) * RS::set_bytes(n);
      return VPM_OK;
    });
  });
}

int vpm_sweep_pairs_partial(int op, const void* records, int64_t n, int64_t tile_begin,
                            int64_t tile_end, int64_t pair_begin, int64_t pair_end,
                            double* rows, int precision, void* workspace,
                            size_t workspace_bytes, void* stream) {
  if (op != VPM_OP_VELOCITY_AND_STRENGTH_GRADIENTS)
    return fail(VPM_ERR_ARG, "pair shards are built for the fused velocity + stretching sum");
  if (n <= 0) return fail(VPM_ERR_ARG, "n must be positive");
  if (!records || !rows || !workspace) return fail(VPM_ERR_ARG, "null pointer");
  if (reinterpret_cast<uintptr_t>(records) % 16 != 0)
    return fail(VPM_ERR_ALIGN, "records must be 16-byte aligned");
  if (reinterpret_cast<uintptr_t>(workspace) % kAlign != 0)
    return fail(VPM_ERR_ALIGN, "workspace must be 256-byte aligned");
  int rc = check_arch();
  if (rc) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  return with_precision(precision, [&](auto P) {
    using Pp = decltype(P);
    return with_fused_both<typename Pp::type, Pp::refine, Pp::uc>(n, [&](auto rs,
                                                                        const Plan& p) {
      using RS = decltype(rs);
      const int64_t nt = RS::tiles(n);
      if (tile_begin < 0 || tile_end < tile_begin || tile_end > nt)
        return fail(VPM_ERR_ARG, "tile range outside [0, " + std::to_string(nt) + ")");
      if (pair_begin < 0 || pair_end < pair_begin || pair_end > nt / 2)
        return fail(VPM_ERR_ARG, "pair range outside [0, " + std::to_string(nt / 2) + ")");
      const size_t need = size_t(RS::sets(p.pairs)) * RS::set_bytes(n);
      if (workspace_bytes < need)
        return fail(VPM_ERR_WORKSPACE, "workspace has " + std::to_string(workspace_bytes) +
                                           " bytes, needs " + std::to_string(need));
      double* acc = static_cast<double*>(workspace);
      int r = RS::launch_part(p, records, n, acc, int(tile_begin), int(tile_end),
                              int(pair_begin) + 1, int(pair_end) + 1, st);
      if (r) return r;
      sets_to_rows_kernel<RS::NV><<<unsigned((n + 255) / 256), 256, 0, st>>>(
          acc, int(RS::sets(p.pairs)), n, rows);
      cudaError_t e = cudaGetLastError();
      return e == cudaSuccess ? VPM_OK : cuda_fail(e, "rows launch");
    });
  });
}

int vpm_finalize_pairs_partial(int op, const double* rows, const void* records,
                               int64_t target_begin, int64_t m, double* out, double* out2,
                               int precision, void* stream) {
  if (op != VPM_OP_VELOCITY_AND_STRENGTH_GRADIENTS)
    return fail(VPM_ERR_ARG, "pair shards are built for the fused velocity + stretching sum");
  if (m < 0 || target_begin < 0) return fail(VPM_ERR_ARG, "negative size or offset");
  if (m == 0) return VPM_OK;
  if (!rows || !records || !out || !out2) return fail(VPM_ERR_ARG, "null pointer");
  if (reinterpret_cast<uintptr_t>(records) % 16 != 0)
    return fail(VPM_ERR_ALIGN, "records must be 16-byte aligned");
  int rc = check_arch();
  if (rc) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  static_assert(OpVelStretchBoth<false, false>::NV == 9 && OpVelStretchBoth64<false>::NV == 9,
                "the fused sum's 9 values per row");
  const unsigned blocks = unsigned((m + 255) / 256);
  switch (precision & ~kPrecisionFlags) {
    case VPM_FP64:
      finalize_rows_kernel<double, FIN_VELSTRETCH, 9><<<blocks, 256, 0, st>>>(
          rows, m, static_cast<const Rec<double>*>(records) + target_begin, out, out2);
      break;
    case VPM_FP32C:
    case VPM_FP32C_REFINED:
      finalize_rows_kernel<float2, FIN_VELSTRETCH, 9><<<blocks, 256, 0, st>>>(
          rows, m, static_cast<const Rec<float2>*>(records) + target_begin, out, out2);
      break;
    default:
      return fail(VPM_ERR_ARG, "unknown precision " + std::to_string(precision));
  }
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? VPM_OK : cuda_fail(e, "finalize launch");
}

int vpm_plan_info(int op, int precision, int64_t m, int64_t n, int64_t* target_blocks,
                  int* splits, int* threads, int* targets_per_thread) {
  if (op == VPM_OP_RHS_VJP || op == VPM_OP_RHS_VJP_PSE || op == VPM_OP_KINETIC_ENERGY_GRAD)
    precision &= ~VPM_UNIFORM_CORE;
  Plan p;
  const int rc = with_precision(precision, [&](auto P) {
    using Pp = decltype(P);
    return plan_op<typename Pp::type, Pp::refine, Pp::uc>(
        op, m, n, &p, (precision & VPM_COMPACT_WORKSPACE) != 0);
  });
  if (rc) return rc;
  if (target_blocks) *target_blocks = p.tblocks;
  if (splits) *splits = p.splits;
  if (threads) *threads = p.threads;
  if (targets_per_thread) *targets_per_thread = p.r;
  return VPM_OK;
}

int vpm_induced_velocity_at(const double* targets, int64_t m, const double* positions,
                            const double* strengths, const double* radii, int64_t n,
                            double* velocities, int precision, void* workspace,
                            size_t workspace_bytes, void* stream) {
  Call c{VPM_OP_INDUCED_VELOCITY_AT, targets, m, positions, strengths, radii, nullptr, n,
         velocities, nullptr, 0, workspace, workspace_bytes, static_cast<cudaStream_t>(stream)};
  return dispatch(c, precision);
}

int vpm_selfinduced_velocity(const double* positions, const double* strengths,
                             const double* radii, int64_t n, double* velocities, int precision,
                             void* workspace, size_t workspace_bytes, void* stream) {
  Call c{VPM_OP_SELFINDUCED_VELOCITY, nullptr, n, positions, strengths, radii, nullptr, n,
         velocities, nullptr, 0, workspace, workspace_bytes, static_cast<cudaStream_t>(stream)};
  return dispatch(c, precision);
}

int vpm_vorticity_field_at(const double* targets, int64_t m, const double* positions,
                           const double* strengths, const double* radii, int64_t n,
                           double* vorticities, int precision, void* workspace,
                           size_t workspace_bytes, void* stream) {
  Call c{VPM_OP_VORTICITY_FIELD_AT, targets, m, positions, strengths, radii, nullptr, n,
         vorticities, nullptr, 0, workspace, workspace_bytes, static_cast<cudaStream_t>(stream)};
  return dispatch(c, precision);
}

int vpm_strength_gradients(const double* positions, const double* strengths,
                           const double* radii, int64_t n, double* dalpha_dt, int precision,
                           void* workspace, size_t workspace_bytes, void* stream) {
  Call c{VPM_OP_STRENGTH_GRADIENTS, nullptr, n, positions, strengths, radii, nullptr, n,
         dalpha_dt, nullptr, 0, workspace, workspace_bytes, static_cast<cudaStream_t>(stream)};
  return dispatch(c, precision);
}

int vpm_strength_gradients_pse(const double* positions, const double* strengths,
                               const double* radii, const double* viscosities, int64_t n,
                               double* dalpha_dt, int precision, void* workspace,
                               size_t workspace_bytes, void* stream) {
  Call c{VPM_OP_STRENGTH_GRADIENTS_PSE, nullptr, n, positions, strengths, radii, viscosities, n,
         dalpha_dt, nullptr, 0, workspace, workspace_bytes, static_cast<cudaStream_t>(stream)};
  return dispatch(c, precision);
}

int vpm_total_kinetic_energy(const double* positions, const double* strengths,
                             const double* radii, int64_t n, double* energy, int precision,
                             void* workspace, size_t workspace_bytes, void* stream) {
  if (!energy) return fail(VPM_ERR_ARG, "null output pointer");
  Call c{VPM_OP_TOTAL_KINETIC_ENERGY, nullptr, n, positions, strengths, radii, nullptr, n,
         energy, nullptr, 0, workspace, workspace_bytes, static_cast<cudaStream_t>(stream)};
  return dispatch(c, precision);
}

int vpm_total_helicity(const double* positions, const double* strengths, const double* radii,
                       int64_t n, int ref_extra_4pi, double* helicity, int precision,
                       void* workspace, size_t workspace_bytes, void* stream) {
  if (!helicity) return fail(VPM_ERR_ARG, "null output pointer");
  Call c{VPM_OP_TOTAL_HELICITY, nullptr, n, positions, strengths, radii, nullptr, n,
         helicity, nullptr, ref_extra_4pi, workspace, workspace_bytes,
         static_cast<cudaStream_t>(stream)};
  return dispatch(c, precision);
}

int vpm_total_enstrophy(const double* positions, const double* strengths, const double* radii,
                        int64_t n, int ref_extra_4pi, double* enstrophy, int precision,
                        void* workspace, size_t workspace_bytes, void* stream) {
  if (!enstrophy) return fail(VPM_ERR_ARG, "null output pointer");
  Call c{VPM_OP_TOTAL_ENSTROPHY, nullptr, n, positions, strengths, radii, nullptr, n,
         enstrophy, nullptr, ref_extra_4pi, workspace, workspace_bytes,
         static_cast<cudaStream_t>(stream)};
  return dispatch(c, precision);
}

int vpm_velocity_and_strength_gradients(const double* positions, const double* strengths,
                                        const double* radii, int64_t n, double* velocities,
                                        double* dalpha_dt, int precision, void* workspace,
                                        size_t workspace_bytes, void* stream) {
  Call c{VPM_OP_VELOCITY_AND_STRENGTH_GRADIENTS, nullptr, n, positions, strengths, radii,
         nullptr, n, velocities, dalpha_dt, 0, workspace, workspace_bytes,
         static_cast<cudaStream_t>(stream)};
  return dispatch(c, precision);
}

int64_t vpm_set_symmetric_min_n(int64_t n) { return g_sym_min_n.exchange(n); }

int64_t vpm_sweep_launches(int op, int precision, int64_t m, int64_t n) {
  if (m <= 0 || n <= 0) return 0;
  if (op == VPM_OP_RHS_VJP || op == VPM_OP_RHS_VJP_PSE || op == VPM_OP_KINETIC_ENERGY_GRAD)
    precision &= ~VPM_UNIFORM_CORE;
  Plan p;
  const int rc = with_precision(precision, [&](auto P) {
    using Pp = decltype(P);
    return plan_op<typename Pp::type, Pp::refine, Pp::uc>(
        op, m, n, &p, (precision & VPM_COMPACT_WORKSPACE) != 0);
  });
  if (rc) return -1;
  if (p.triangle) {  // zero the diagonal tiles' sets, those tiles, the triangle, finalize
    return op == VPM_OP_LES_STEP_SUMS ? 5 : 4;
  }
  if (p.pairs) {  // zero the accumulators, the diagonal tiles, the diagonal-pair launches, finalize
    const int64_t npairs = p.tblocks / 2;
    return 3 + (npairs + p.pairs - 1) / p.pairs;
  }
  if (p.circle) return op == VPM_OP_LES_STEP_SUMS ? 3 : 2;
  if (p.small) return 1;  // pack, sweep and finalize in one
  return 2;  // sweep, finalize (or the single-block reduction of a scalar)
}

int vpm_les_step_sums(const double* positions, const double* strengths, const double* radii,
                      int64_t n, double* velocities, double* dalpha_dt, double* vorticity,
                      double* enstrophy, int ref_extra_4pi, int precision, void* workspace,
                      size_t workspace_bytes, void* stream) {
  Call c{VPM_OP_LES_STEP_SUMS, nullptr, n, positions, strengths, radii,
         nullptr, n, velocities, dalpha_dt, ref_extra_4pi, workspace, workspace_bytes,
         static_cast<cudaStream_t>(stream)};
  c.out3 = vorticity;
  c.out4 = enstrophy;
  return dispatch(c, precision);
}

int vpm_les_test_filter(const double* positions, const double* strengths,
                        const double* test_radii, const double* fields, int64_t n,
                        double* test_vorticity, double* test_filtered, int precision,
                        void* workspace, size_t workspace_bytes, void* stream) {
  if (n < 0) return fail(VPM_ERR_ARG, "negative size");
  if (n > 0 && (!positions || !strengths || !test_radii || !fields || !test_vorticity ||
                !test_filtered))
    return fail(VPM_ERR_ARG, "null pointer");
  Call c{VPM_OP_LES_TEST_FILTER, nullptr, n, positions, strengths, test_radii, nullptr, n,
         test_vorticity, test_filtered, 0, workspace, workspace_bytes,
         static_cast<cudaStream_t>(stream)};
  c.aux = fields;
  c.compact = (precision & VPM_COMPACT_WORKSPACE) != 0;
  switch (precision & ~kPrecisionFlags) {
    case VPM_FP64:
      return run_filter<double, false>(c);
    case VPM_FP32C:
      return run_filter<float2, false>(c);
    case VPM_FP32C_REFINED:
      return run_filter<float2, true>(c);
    default:
      return fail(VPM_ERR_ARG, "unknown precision " + std::to_string(precision));
  }
}

size_t vpm_record_bytes(int precision) {
  switch (precision & ~kPrecisionFlags) {
    case VPM_FP64:
      return sizeof(Rec<double>);
    case VPM_FP32C:
    case VPM_FP32C_REFINED:
      return sizeof(Rec<float2>);
    default:
      fail(VPM_ERR_ARG, "unknown precision");
      return 0;
  }
}

int vpm_pack_records(const double* positions, const double* strengths, const double* radii,
                     const double* viscosities, int64_t n, int precision, void* records,
                     void* stream) {
  if (n < 0) return fail(VPM_ERR_ARG, "negative size");
  if (n > 0 && (!positions || !strengths || !radii || !records))
    return fail(VPM_ERR_ARG, "null pointer");
  if (reinterpret_cast<uintptr_t>(records) % 16 != 0)
    return fail(VPM_ERR_ALIGN, "records must be 16-byte aligned");
  int rc = check_arch();
  if (rc) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool uc = (precision & VPM_UNIFORM_CORE) != 0;
  precision &= ~kPrecisionFlags;
  if (precision == VPM_FP64)
    return pack<double>(positions, strengths, radii, viscosities, n,
                        static_cast<Rec<double>*>(records), st, uc);
  if (precision == VPM_FP32C || precision == VPM_FP32C_REFINED)
    return pack<float2>(positions, strengths, radii, viscosities, n,
                        static_cast<Rec<float2>*>(records), st, uc);
  return fail(VPM_ERR_ARG, "unknown precision");
}

int vpm_sweep_records(int op, const void* records, int64_t n, int64_t target_begin, int64_t m,
                      int ref_extra_4pi, double* out, double* out2, int precision,
                      void* workspace, size_t workspace_bytes, void* stream) {
  Call c{op, nullptr, m, nullptr, nullptr, nullptr, nullptr, n, out, out2, ref_extra_4pi,
         workspace, workspace_bytes, static_cast<cudaStream_t>(stream)};
  c.records = records;
  c.tgt_begin = target_begin;
  if (n > 0 && !records) return fail(VPM_ERR_ARG, "null records pointer");
  return dispatch(c, precision);
}

int vpm_rhs_vjp(const double* positions, const double* strengths, const double* radii,
                const double* viscosities, int64_t n, const double* grad_velocities,
                const double* grad_rates, double* grad_positions, double* grad_strengths,
                double* grad_radii, double* grad_viscosities, int precision, void* workspace,
                size_t workspace_bytes, void* stream) {
  GradCall c{viscosities ? VPM_OP_RHS_VJP_PSE : VPM_OP_RHS_VJP, positions, strengths, radii,
             viscosities, grad_velocities, grad_rates, n, grad_positions, grad_strengths,
             grad_radii, grad_viscosities, workspace, workspace_bytes,
             static_cast<cudaStream_t>(stream)};
  return dispatch_grad(c, precision);
}

int vpm_kinetic_energy_grad(const double* positions, const double* strengths,
                            const double* radii, int64_t n, double* grad_positions,
                            double* grad_strengths, double* grad_radii, int precision,
                            void* workspace, size_t workspace_bytes, void* stream) {
  GradCall c{VPM_OP_KINETIC_ENERGY_GRAD, positions, strengths, radii, nullptr, nullptr, nullptr,
             n, grad_positions, grad_strengths, grad_radii, nullptr, workspace,
             workspace_bytes, static_cast<cudaStream_t>(stream)};
  return dispatch_grad(c, precision);
}

// Self-induced velocity without any allocation: the scratch (packed records and per-split
// partial sums) lives in the library's static device array.  Every call shares that array
// and leaves its contents behind; nothing in it needs clearing, because each call that
// completes rewrites every record and partial it reads.  A sweep whose bounded wait gives up
// returns without writing its partials: the call's output is then built from what the
// previous call left, and only the device error word (vpm_device_errors) shows it.  Calls
// that overlap on the GPU (two streams, two host threads) race on the array.  The first call
// in a context looks up the array's address there (cudaGetSymbolAddress) and the kernels'
// occupancy; make that first call before any stream capture.
int vpm_selfinduced_velocity_noalloc(const double* positions, const double* strengths,
                                     const double* radii, int64_t n, double* velocities,
                                     int precision, void* stream) {
  if (n < 0) return fail(VPM_ERR_ARG, "negative size");
  if (n > kNoAllocMaxN)
    return fail(VPM_ERR_ARG, "n = " + std::to_string(n) +
                                 " exceeds the no-allocation limit of " +
                                 std::to_string(kNoAllocMaxN) +
                                 " particles; call vpm_selfinduced_velocity with a workspace");
  int rc = check_arch();
  if (rc) return rc;
  void* scratch = nullptr;
  rc = noalloc_scratch(&scratch);
  if (rc) return rc;
  Call c{VPM_OP_SELFINDUCED_VELOCITY, nullptr, n, positions, strengths, radii, nullptr, n,
         velocities, nullptr, 0, scratch, kNoAllocScratchBytes,
         static_cast<cudaStream_t>(stream)};
  c.max_partial_bytes = kNoAllocScratchBytes - kNoAllocRecordBytes;
  return dispatch(c, precision);
}

int vpm_selftest_bounded_wait(int* timed_out, void* stream) {
  if (!timed_out) return fail(VPM_ERR_ARG, "null result pointer");
  int rc = check_arch();
  if (rc) return rc;
  bounded_wait_selftest_kernel<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(timed_out);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? VPM_OK : cuda_fail(e, "selftest launch");
}

int vpm_launch_fma_peak(int fp64, int blocks, int threads, int iters, void* sink, void* stream) {
  if (blocks <= 0 || threads <= 0 || threads > 1024 || iters <= 0 || !sink || fp64 < 0 ||
      fp64 > 4)
    return fail(VPM_ERR_ARG, "bad fma peak launch arguments");
  int rc = check_arch();
  if (rc) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (fp64 == 4)
    ffma_mixed_peak_kernel<<<blocks, threads, 0, st>>>(iters, static_cast<float*>(sink));
  else if (fp64 == 3)
    ffma2_peak_kernel<<<blocks, threads, 0, st>>>(iters, static_cast<float*>(sink));
  else if (fp64 == 2)
    rsqrt_peak_kernel<<<blocks, threads, 0, st>>>(iters, static_cast<float*>(sink));
  else if (fp64)
    fma_peak_kernel<double><<<blocks, threads, 0, st>>>(iters, static_cast<double*>(sink));
  else
    fma_peak_kernel<float><<<blocks, threads, 0, st>>>(iters, static_cast<float*>(sink));
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? VPM_OK : cuda_fail(e, "fma peak launch");
}

}  // extern "C"

// Element-wise time-step kernels and O(N) diagnostics (same translation unit).
#include "vpm_step.cuh"

// Initial conditions and particle lattices on the device.
#include "vpm_ic.cuh"
