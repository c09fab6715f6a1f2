// Included by the resident_bicgstab_*d.cu that instantiate the launches.
#pragma once

#include "resident_bands.cuh"

namespace cfdb {
namespace res {
namespace {

template <int DIM, int NC, bool PREC>
__global__ void __launch_bounds__(kClusterThreads, 1)
    bicgstab_cluster(BandOp<DIM> A, uint32_t n, uint32_t len, FastDiv dlen, Io P) {
  extern __shared__ __align__(16) double sm[];
  __shared__ TeamSmem ts;
  auto team = cluster_team<kClusterThreads>(&ts, len, dlen);
  bicgstab_run<kClusterThreads, NC, true, PREC>(A, n, len, P, team, sm);
}

template <int DIM, int NC, bool PREC, bool XS>
__global__ void __launch_bounds__(kClusterThreads, 1)
    bicgstab_grid(BandOp<DIM> A, uint32_t n, uint32_t len, GridWords w, Io P) {
  extern __shared__ __align__(16) double sm[];
  __shared__ TeamSmem ts;
  auto team = grid_team<kClusterThreads>(&ts, w);
  bicgstab_run<kClusterThreads, NC, XS, PREC>(A, n, len, P, team, sm);
}

// Runs f for the kernel with a thread's coefficients in registers (one or two
// cells each) or the general one (0).
template <class F>
cudaError_t with_cells(int nc, F f) {
  if (nc == 1) return f(std::integral_constant<int, 1>{});
  if (nc == 2) return f(std::integral_constant<int, 2>{});
  return f(std::integral_constant<int, 0>{});
}

}  // namespace

template <int DIM>
int bicgstab_cluster_limit() {
  return cluster_limit((const void*)bicgstab_cluster<DIM, 0, true>, kClusterThreads);
}

template <int DIM, bool PREC>
cudaError_t launch_bicgstab(cfdb_context* ctx, const BandOp<DIM>& A, const Plan& P, uint32_t n,
                            const GridWords& w, const Io& io) {
  if (P.team == 1)
    return with_cells(P.nc, [&](auto nc) {
      auto fn = bicgstab_cluster<DIM, decltype(nc)::value, PREC>;
      if (cluster_limit((const void*)fn, kClusterThreads) < P.blocks) return cudaErrorInvalidConfiguration;
      return launch_cluster(fn, P.blocks, P.blocks, kClusterThreads, P.smem, ctx->stream, A, n, P.len,
                            fast_div(P.len), io);
    });
  return with_cells(P.nc, [&](auto nc) {
    constexpr int NC = decltype(nc)::value;
    const void* fn = (const void*)bicgstab_grid<DIM, NC, PREC, true>;
    if constexpr (NC == 0)  // x of one or two cells a thread always fits
      if (!P.xs) fn = (const void*)bicgstab_grid<DIM, NC, PREC, false>;
    return cooperative<DIM>(fn, P, ctx->stream, A, n, w, io);
  });
}

}  // namespace res
}  // namespace cfdb
