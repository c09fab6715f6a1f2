// The stencil Krylov solves (BiCGSTAB, CG, optional Jacobi) with their
// vectors on chip (resident.cuh), for the systems that fit.
#include <cuda_runtime.h>

#include <type_traits>

#include "resident_launch.cuh"
#include "stencil_solve.cuh"

namespace cfdb {
namespace {

using namespace res;

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

template <int DIM>
cudaError_t cooperative(const void* fn, const Plan& P, cudaStream_t st, BandOp<DIM> A, uint32_t n,
                        GridWords w, Io io) {
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
  if (e != cudaSuccess) return e;
  uint32_t len = P.len;
  void* args[] = {&A, &n, &len, &w, &io};
  return cudaLaunchCooperativeKernel(fn, dim3(P.blocks), dim3(P.threads), args, P.smem, st);
}

// Runs f for the kernel with a thread's coefficients in registers (one or two
// cells each) or the general one (0).
template <class F>
cudaError_t with_cells(int nc, F f) {
  if (nc == 1) return f(std::integral_constant<int, 1>{});
  if (nc == 2) return f(std::integral_constant<int, 2>{});
  return f(std::integral_constant<int, 0>{});
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
    const void* fn = P.xs ? (const void*)bicgstab_grid<DIM, NC, PREC, true>
                          : (const void*)bicgstab_grid<DIM, NC, PREC, false>;
    return cooperative<DIM>(fn, P, ctx->stream, A, n, w, io);
  });
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
    const void* fn = P.halo ? (P.xs ? (const void*)cg_grid<DIM, T, NC, true, true>
                                    : (const void*)cg_grid<DIM, T, NC, false, true>)
                            : (P.xs ? (const void*)cg_grid<DIM, T, NC, true, false>
                                    : (const void*)cg_grid<DIM, T, NC, false, false>);
    return cooperative<DIM>(fn, P, ctx->stream, A, n, w, io);
  };
  if (P.threads == kGridThreadsSmall)
    return with_nc(P.nc, SmallNCs{}, [&](auto nc) { return go(std::integral_constant<int, kGridThreadsSmall>{}, nc); });
  return with_nc(P.nc, LargeNCs{}, [&](auto nc) { return go(std::integral_constant<int, kGridThreadsLarge>{}, nc); });
}

template <int DIM>
cfdb_status run(cfdb_context* ctx, const StencilMatrix& M, int krylov, const Io& io, bool* taken) {
  *taken = false;
  const int limit = krylov == 1
                        ? cluster_limit((const void*)bicgstab_cluster<DIM, 0, true>, kClusterThreads)
                        : cluster_limit((const void*)cg_cluster<DIM, 8>, kClusterThreads);
  const BandOp<DIM> A = band_op<DIM>(M);
  const Plan P = krylov == 1 ? bicgstab_plan(M.n, ctx->num_sms, limit)
                             : cg_plan(M.n, A.sz, ctx->num_sms, limit);
  if (P.team == 0) return CFDB_OK;
  *taken = true;
  GridWords w;
  cfdb_status st = prepare_words(ctx, P, &w);
  if (st != CFDB_OK) return st;
  CFDB_CUDA(ctx, cudaEventRecord(ctx->ev_k0, ctx->stream));
  const uint32_t n = (uint32_t)M.n;
  const cudaError_t e = krylov == 1 ? (M.inv ? launch_bicgstab<DIM, true>(ctx, A, P, n, w, io)
                                             : launch_bicgstab<DIM, false>(ctx, A, P, n, w, io))
                                    : launch_cg<DIM>(ctx, A, P, n, w, io);
  if (e != cudaSuccess) return cuda_error(ctx, e, "on-chip Krylov launch", __FILE__, __LINE__);
  CFDB_CUDA(ctx, cudaEventRecord(ctx->ev_k1, ctx->stream));
  return CFDB_OK;
}

}  // namespace

cfdb_status resident_stencil_solve(cfdb_context* ctx, const StencilMatrix& M, StencilWork& W,
                                   const double* b, double* x, int krylov, double abs_tol,
                                   double rel_tol, int64_t max_it, double* hist, int64_t hist_cap,
                                   bool* taken) {
  Io io{};
  io.b = b;
  io.x = x;
  io.pub = W.p;
  io.pub2 = W.s;
  io.abs_tol = abs_tol;
  io.rel_tol = rel_tol;
  io.max_it = max_it;
  io.hist = hist;
  io.hist_cap = hist_cap;
  io.out = ctx->scalars;
  return M.dim == 2 ? run<2>(ctx, M, krylov, io, taken) : run<3>(ctx, M, krylov, io, taken);
}

}  // namespace cfdb
