// Included by the resident_cg_*d.cu that instantiate the launches.
#pragma once

#include "resident_bands.cuh"

namespace cfdb {
namespace res {
namespace {

template <int DIM, int NC>
__global__ void __launch_bounds__(kClusterThreads, 1)
    cg_cluster(BandOp<DIM> A, uint32_t n, uint32_t len, FastDiv dlen, Io P) {
  extern __shared__ __align__(16) double sm[];
  __shared__ TeamSmem ts;
  auto team = cluster_team<kClusterThreads>(&ts, len, dlen);
  cg_run<kClusterThreads, NC, (NC <= 2), true, true>(A, n, len, P, team, sm);
}

template <int DIM, int T, int NC, bool XS, bool HALO>
__global__ void __launch_bounds__(T, 1)
    cg_grid(BandOp<DIM> A, uint32_t n, uint32_t len, GridWords w, Io P) {
  extern __shared__ __align__(16) double sm[];
  __shared__ TeamSmem ts;
  auto team = grid_team<T>(&ts, w);
  cg_run<T, NC, false, XS, HALO>(A, n, len, P, team, sm);
}

using ClusterNCs = std::integer_sequence<int, 1, 2, 3, 4, 6, 8>;
using SmallNCs = std::integer_sequence<int, 1, 2, 4>;
using LargeNCs = std::integer_sequence<int, 4, 8, 14>;

}  // namespace

template <int DIM>
int cg_cluster_limit() {
  return cluster_limit((const void*)cg_cluster<DIM, 8>, kClusterThreads);
}

template <int DIM>
cudaError_t launch_cg(cfdb_context* ctx, const BandOp<DIM>& A, const Plan& P, uint32_t n,
                      const GridWords& w, const Io& io) {
  if (P.team == 1)
    return with_nc(P.nc, ClusterNCs{}, [&](auto nc) {
      auto fn = cg_cluster<DIM, decltype(nc)::value>;
      if (cluster_limit((const void*)fn, kClusterThreads) < P.blocks) return cudaErrorInvalidConfiguration;
      return launch_cluster(fn, P.blocks, P.blocks, kClusterThreads, P.smem, ctx->stream, A, n, P.len,
                            fast_div(P.len), io);
    });
  auto go = [&](auto threads, auto nc) {
    constexpr int T = decltype(threads)::value, NC = decltype(nc)::value;
    const void* fn = P.halo ? (const void*)cg_grid<DIM, T, NC, true, true>
                            : (const void*)cg_grid<DIM, T, NC, true, false>;
    if constexpr (T == kGridThreadsLarge) {  // a small block's x always fits (cg_plan)
      if (!P.xs && P.halo) fn = (const void*)cg_grid<DIM, T, NC, false, true>;
      // alone, p, r and x leave the block's memory only at the most cells a thread
      if constexpr ((size_t)3 * NC * T * sizeof(double) > kSmemMax)
        if (!P.xs && !P.halo) fn = (const void*)cg_grid<DIM, T, NC, false, false>;
    }
    return cooperative<DIM>(fn, P, ctx->stream, A, n, w, io);
  };
  if (P.threads == kGridThreadsSmall)
    return with_nc(P.nc, SmallNCs{}, [&](auto nc) { return go(std::integral_constant<int, kGridThreadsSmall>{}, nc); });
  return with_nc(P.nc, LargeNCs{}, [&](auto nc) { return go(std::integral_constant<int, kGridThreadsLarge>{}, nc); });
}

}  // namespace res
}  // namespace cfdb
