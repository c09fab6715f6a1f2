// The FP64 Jacobi-PCG of the p' operator with its vectors on chip
// (resident.cuh): the systems that fit one thread-block cluster, or the
// shared memory of the whole GPU.
#include <cuda_runtime.h>

#include <type_traits>

#include "pcg_internal.cuh"
#include "resident_launch.cuh"

namespace cfdb {
namespace {

using namespace res;

template <int DIM, int NC>
__global__ void __launch_bounds__(kClusterThreads, 1)
    pcg_cluster(FaceOp<DIM> A, uint32_t n, uint32_t len, FastDiv dlen, Io P) {
  extern __shared__ __align__(16) double sm[];
  __shared__ TeamSmem ts;
  auto T = cluster_team<kClusterThreads>(&ts, len, dlen);
  cg_run<kClusterThreads, NC, (NC <= 2), true, true>(A, n, len, P, T, sm);
}

template <int DIM, int T, int NC, bool XS, bool HALO>
__global__ void __launch_bounds__(T, 1)
    pcg_grid(FaceOp<DIM> A, uint32_t n, uint32_t len, GridWords w, Io P) {
  extern __shared__ __align__(16) double sm[];
  __shared__ TeamSmem ts;
  auto team = grid_team<T>(&ts, w);
  cg_run<T, NC, false, XS, HALO>(A, n, len, P, team, sm);
}

using ClusterNCs = std::integer_sequence<int, 1, 2, 3, 4, 6, 8>;
using SmallNCs = std::integer_sequence<int, 1, 2, 4>;
using LargeNCs = std::integer_sequence<int, 4, 8, 14>;

template <int DIM>
cfdb_status run(cfdb_context* ctx, const OpView<double>& V, const double* invd, const Plan& P,
                uint32_t n, const Io& io) {
  FaceOp<DIM> A{};
  A.A = V;
  A.invd = invd;
  A.nx = V.nx;
  A.ny = V.ny;
  A.nz = V.nz;
  A.sz = (uint32_t)V.nx * V.ny;
  A.dx = fast_div(V.nx);
  A.dy = fast_div(V.ny);
  GridWords w;
  cfdb_status st = prepare_words(ctx, P, &w);
  if (st != CFDB_OK) return st;
  CFDB_CUDA(ctx, cudaEventRecord(ctx->ev_k0, ctx->stream));
  cudaError_t e;
  if (P.team == 1) {
    e = with_nc(P.nc, ClusterNCs{}, [&](auto nc) {
      auto fn = pcg_cluster<DIM, decltype(nc)::value>;
      if (cluster_limit((const void*)fn, kClusterThreads) < P.blocks) return cudaErrorInvalidConfiguration;
      return launch_cluster(fn, P.blocks, P.blocks, kClusterThreads, P.smem, ctx->stream, A, n, P.len,
                            fast_div(P.len), io);
    });
  } else {
    auto go = [&](auto threads, auto nc) {
      constexpr int T = decltype(threads)::value, NC = decltype(nc)::value;
      const void* fn = P.halo ? (P.xs ? (const void*)pcg_grid<DIM, T, NC, true, true>
                                      : (const void*)pcg_grid<DIM, T, NC, false, true>)
                              : (P.xs ? (const void*)pcg_grid<DIM, T, NC, true, false>
                                      : (const void*)pcg_grid<DIM, T, NC, false, false>);
      cudaError_t q = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
      if (q != cudaSuccess) return q;
      FaceOp<DIM> a = A;
      uint32_t nn = n, len = P.len;
      Io o = io;
      void* args[] = {&a, &nn, &len, &w, &o};
      return cudaLaunchCooperativeKernel(fn, dim3(P.blocks), dim3(T), args, P.smem, ctx->stream);
    };
    if (P.threads == kGridThreadsSmall)
      e = with_nc(P.nc, SmallNCs{}, [&](auto nc) { return go(std::integral_constant<int, kGridThreadsSmall>{}, nc); });
    else
      e = with_nc(P.nc, LargeNCs{}, [&](auto nc) { return go(std::integral_constant<int, kGridThreadsLarge>{}, nc); });
  }
  if (e != cudaSuccess) return cuda_error(ctx, e, "on-chip PCG launch", __FILE__, __LINE__);
  CFDB_CUDA(ctx, cudaEventRecord(ctx->ev_k1, ctx->stream));
  count_launch(ctx);
  return CFDB_OK;
}

}  // namespace

bool resident_pcg_fits(const cfdb_context* ctx, const OpView<double>& A) {
  return cg_plan((int64_t)A.nx * A.ny * A.nz, (int64_t)A.nx * A.ny, ctx->num_sms, 0).team != 0;
}

cfdb_status resident_pcg(cfdb_context* ctx, const OpView<double>& A, int dim, const double* invd,
                         const double* b, double* x, double* pub, double* inv,
                         double abs_tol, double rel_tol,
                         int64_t max_it, double* hist, int64_t hist_cap) {
  const int64_t n = (int64_t)A.nx * A.ny * A.nz;
  const int limit = dim == 2 ? cluster_limit((const void*)pcg_cluster<2, 8>, kClusterThreads)
                             : cluster_limit((const void*)pcg_cluster<3, 8>, kClusterThreads);
  const Plan P = cg_plan(n, (int64_t)A.nx * A.ny, ctx->num_sms, limit);
  Io io{};
  io.b = b;
  io.x = x;
  io.pub = pub;
  io.inv = inv;
  io.abs_tol = abs_tol;
  io.rel_tol = rel_tol;
  io.max_it = max_it;
  io.hist = hist;
  io.hist_cap = hist_cap;
  io.out = ctx->scalars;
  return dim == 2 ? run<2>(ctx, A, invd, P, (uint32_t)n, io) : run<3>(ctx, A, invd, P, (uint32_t)n, io);
}

}  // namespace cfdb
