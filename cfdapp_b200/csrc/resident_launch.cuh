// Choice and launch of the on-chip Krylov kernels (resident.cuh).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include "cfdb_internal.cuh"
#include "resident.cuh"

namespace cfdb {
namespace res {

constexpr unsigned long long kTimeoutNs = 2000000000ull;
constexpr size_t kSmemMax = 225 * 1024;  // of the 227 KB a block may have, beside TeamSmem
constexpr int kClusterThreads = 512;
constexpr int kClusterNC = 8, kGridNC = 14;  // most cells per thread
// Threads of a grid team's blocks: 1024 once every thread has several cells
// (a reduction over 512 threads is 0.5 us faster).
constexpr int kGridThreadsSmall = 512, kGridThreadsLarge = 1024;
constexpr uint32_t kGridSmallCells = 2048;  // cells per block

// As cluster_cells; a BiCGSTAB iteration (us, cluster / grid): 129^2 12.2 / 13,
// 181^2 13.4 / 13.5, 33^3 16.7 / 17.
constexpr int64_t kBicgClusterCells = 32768;

struct Plan {
  int team = 0;  // 0: does not fit; 1: one cluster; 2: the grid
  int blocks = 0;
  uint32_t len = 0;
  int nc = 0;
  bool xs = false;    // x in shared memory too
  int threads = 0;
  bool halo = false;  // p of the neighbouring planes kept in shared memory
  size_t smem = 0;
};

// Cells a cluster takes before the whole GPU is the faster team, by the time
// of an FP64 CG iteration (us, cluster / grid).  2D: 150^2 4.9 / 5.9, 181^2
// (32 761 cells: the last with four a thread) 5.65 / 5.92, 182^2 6.05 / 5.74,
// 190^2 6.11 / 5.76.  3D, whose ranges read larger planes: 26^3 5.4 / 6.2,
// 29^3 6.1 / 6.4, 30^3 6.7 / 6.4, 33^3 7.3 / 6.3.  (Mixed precision meets at
// the same places within 5 %.)
constexpr int64_t cluster_cells(int dim) { return dim == 2 ? 32768 : 25600; }

// Layout of the CG of n cells.  A cluster's size grows with the system until every
// block has one cell per thread; per iteration (us, streaming kernel before):
// 40x33 2.7 (18.6), 129^2 4.7 (13.0), 512^2 8.0 (20.9), 64^3 9.6 (19.5),
// 96^3 16.7 (29.3), 128^3 31.8 (44.7); the last two keep no neighbouring
// planes.  `reach`: cells the stencil reaches (a plane); max_cluster: 0 past
// cluster_cells.
inline Plan cg_plan(int64_t n, int64_t reach, int num_sms, int max_cluster, size_t word = 8) {
  Plan P;
  auto fill = [&](int team, int blocks, int max_nc, bool halo) {
    P = Plan{};
    P.len = (uint32_t)((n + blocks - 1) / blocks);
    const int threads = team == 1 ? kClusterThreads
                                  : (P.len <= kGridSmallCells ? kGridThreadsSmall : kGridThreadsLarge);
    P.threads = threads;
    P.blocks = team == 1 ? blocks : (int)((n + P.len - 1) / P.len);
    P.nc = (int)((P.len + threads - 1) / threads);
    P.halo = halo;
    const size_t words = (size_t)P.len * (team == 1 ? 3 : 2) + (halo ? 2 * (size_t)reach : 0);
    P.xs = (words + P.len) * word <= kSmemMax;
    P.smem = (words + (P.xs ? P.len : 0)) * word;
    // a cluster's kernel and that of few cells a block have x in shared memory
    // always (the latter fits without the neighbouring planes)
    if (P.nc <= max_nc && P.smem <= kSmemMax && (threads == kGridThreadsLarge || P.xs)) P.team = team;
  };
  if (max_cluster > 0) {
    int blocks = 1;
    while (blocks < max_cluster && (int64_t)blocks * kClusterThreads < n) blocks *= 2;
    fill(1, blocks, kClusterNC, true);
  }
  if (!P.team) fill(2, num_sms, kGridNC, true);
  if (!P.team) fill(2, num_sms, kGridNC, false);
  return P;
}

// Layout of the BiCGSTAB of n cells: p, r, rHat, v, t (and x) in shared memory.
inline Plan bicgstab_plan(int64_t n, int num_sms, int max_cluster) {
  Plan P;
  auto fill = [&](int team, int blocks) {
    P = Plan{};
    P.len = (uint32_t)((n + blocks - 1) / blocks);
    P.blocks = team == 1 ? blocks : (int)((n + P.len - 1) / P.len);
    P.threads = kClusterThreads;
    P.nc = (int)((P.len + P.threads - 1) / P.threads);
    P.xs = (size_t)6 * P.len * 8 <= kSmemMax;
    P.smem = (size_t)(P.xs ? 6 : 5) * P.len * 8;
    if (P.smem <= kSmemMax && (team == 2 || P.xs)) P.team = team;
  };
  if (n <= kBicgClusterCells && max_cluster > 0) {
    int blocks = 1;
    while (blocks < max_cluster && (int64_t)blocks * kClusterThreads < n) blocks *= 2;
    fill(1, blocks);
  }
  if (!P.team) fill(2, num_sms);
  return P;
}

// Shared memory of one cluster of kMaxCluster blocks running the CG or the
// BiCGSTAB of n cells with everything in shared memory; 0: does not fit.
inline size_t cluster_smem(int64_t n, int64_t reach, int krylov, int max_nc) {
  const size_t len = (size_t)((n + kMaxCluster - 1) / kMaxCluster);
  const size_t words = krylov == 1 ? 6 * len : 4 * len + 2 * (size_t)reach;
  if (words * 8 > kSmemMax || len > (size_t)max_nc * kClusterThreads) return 0;
  return words * 8;
}

// Whether clusters of kMaxCluster blocks, one per case and kClustersAtOnce at
// a time, end the solves of a batch sooner than block teams, which advance
// all cases together.  side, cells: each case's longest side and cells.
//
// A solve's iterations: in proportion to its side for the p' systems
// (poisson), alike for the diagonally dominant momentum systems.  The time of
// an iteration, as a share of a team's in a small batch (about 25 us), from
// solves of 4 to 64 equal cases:
//   cluster  CG 0.2 up to 2 cells a thread (48^2 0.20, 128^2 0.18), then 0.33
//            (192^2; 33^3 0.28) to 0.41 (256^2); BiCGSTAB 0.31 (128^2 0.30), 0.39, 0.46
//   teams    1 until the batch's vectors fill L2, then in proportion to its
//            cells: 1.2 at 0.85 M, 1.4 at 1.05 M, 2.4 at 1.8 M, 3.2 at 2.4 M
// p' solves of an outer iteration (ms, clusters / teams): 128^2 x 16 9.4 /
// 17.7, x 32 15.6 / 18.6, x 48 21.9 / 20.0, x 64 31.1 / 22.9; 48^2 x 64 9.7 /
// 4.9; 256^2 x 32 67.5 / 99.4.  Momentum: 48^2 x 16 1.19 / 1.18, x 64 4.0 /
// 1.2; 256^2 x 16 1.9 / 2.2.
constexpr int kClustersAtOnce = 7;
inline bool clusters_pay(int dim, int ncases, const int64_t* side, const int64_t* cells, int krylov,
                         bool poisson) {
  double all = 0.0, longest = 0.0;
  double busy[kClustersAtOnce] = {};
  std::vector<double> cost(ncases);
  for (int k = 0; k < ncases; ++k) {
    const double its = poisson ? (double)side[k] : 1.0, n = (double)cells[k];
    const bool few = cells[k] <= 2 * kMaxCluster * kClusterThreads;
    const double cg = few ? 0.2 : (0.23 + 2.8e-6 * n) * (dim == 3 ? 0.85 : 1.0);
    cost[k] = its * (krylov == 1 ? (few ? 0.31 : 0.30 + 2.5e-6 * n) : cg);
    all += n;
    longest = std::max(longest, its);
  }
  const double teams = longest * std::max(1.0 + 0.24e-6 * all, 1.35e-6 * all);
  std::sort(cost.begin(), cost.end(), [](double a, double b) { return a > b; });
  for (double c : cost) *std::min_element(busy, busy + kClustersAtOnce) += c;
  return *std::max_element(busy, busy + kClustersAtOnce) < teams;
}

// Largest cluster size (16, 8, ... 1; 0 on failure) `fn` can run at with the
// most shared memory, and its opt-ins, once per kernel and device.
inline int cluster_limit(const void* fn, int threads) {
  static std::mutex mu;
  static std::map<std::pair<const void*, int>, int> cache;
  std::lock_guard<std::mutex> lock(mu);
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  auto it = cache.find({fn, dev});
  if (it != cache.end()) return it->second;
  int best = 0;
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax) == cudaSuccess &&
      cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
    for (int c = kMaxCluster; c >= 1 && !best; c /= 2) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = c;
      cfg.blockDim = threads;
      cfg.dynamicSmemBytes = kSmemMax;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = c;
      at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int num = 0;
      if (cudaOccupancyMaxActiveClusters(&num, fn, &cfg) == cudaSuccess && num >= 1) best = c;
      else cudaGetLastError();
    }
  }
  cudaGetLastError();
  return cache[{fn, dev}] = best;
}

template <typename... KArgs, typename... Args>
cudaError_t launch_cluster(void (*kernel)(KArgs...), int blocks, int cluster, int threads,
                           size_t smem, cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = blocks;
  cfg.blockDim = threads;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = cluster;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

struct GridWords {
  double* partials;
  unsigned* count;
  unsigned* error;
};

template <int THREADS>
__device__ __forceinline__ ClusterTeam<THREADS> cluster_team(TeamSmem* ts, uint32_t len, FastDiv dlen) {
  ClusterTeam<THREADS> T;
  uint32_t r, s;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(s));
  T.rank_ = (int)r;
  T.size_ = (int)s;
  T.len = len;
  T.dlen = dlen;
  T.ts = ts;
  return T;
}

template <int THREADS>
__device__ __forceinline__ GridTeam<THREADS> grid_team(TeamSmem* ts, const GridWords& w) {
  GridTeam<THREADS> T;
  T.partials = w.partials;
  T.count = w.count;
  T.error = w.error;
  T.timeout_ns = kTimeoutNs;
  T.rank_ = blockIdx.x;
  T.size_ = gridDim.x;
  T.ts = ts;
  return T;
}

// Runs f(std::integral_constant NC) for the smallest instantiated NC >= nc.
template <int... NCS, class F>
cudaError_t with_nc(int nc, std::integer_sequence<int, NCS...>, F f) {
  cudaError_t e = cudaErrorInvalidValue;
  bool done = false;
  ((!done && nc <= NCS ? (done = true, e = f(std::integral_constant<int, NCS>{})) : e), ...);
  return e;
}

// Zeroes the barrier words and the outcome scalars.
inline cfdb_status prepare_words(cfdb_context* ctx, const Plan& P, GridWords* w) {
  if (P.team == 2) {
    cfdb_status st = ensure_partials(ctx, (size_t)2 * P.blocks * kMaxVals);
    if (st != CFDB_OK) return st;
  }
  w->partials = ctx->partials;
  w->count = ctx->sync_words;
  w->error = ctx->sync_words + 2;
  CFDB_CUDA(ctx, cudaMemsetAsync(ctx->sync_words, 0, 4 * sizeof(unsigned), ctx->stream));
  CFDB_CUDA(ctx, cudaMemsetAsync(ctx->scalars, 0, 8 * sizeof(double), ctx->stream));
  return CFDB_OK;
}

}  // namespace res
}  // namespace cfdb
