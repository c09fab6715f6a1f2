// The Jacobi-PCG of the p' operator with its vectors on chip (resident.cuh):
// the systems that fit one thread-block cluster, or the shared memory of the
// whole GPU.  FP64, mixed precision (FP32 directions) and FP32 (the inner
// solves of the refinement form).  A mixed solve (us per iteration, streaming
// kernel before): 128^2 3.8 (18.3), 64^3 10.6 (19.1), 96x80x64 14.5 (27.7),
// 128^3 34.3 (43.2); a refinement's FP32 iteration: 130x128 4.8 (12.0),
// 65x60x50 9.7 (24.3), 127x120x100 24.2 (61.9).
#include <cuda_runtime.h>

#include <type_traits>

#include "pcg_internal.cuh"
#include "resident_launch.cuh"

namespace cfdb {
namespace {

using namespace res;

enum { FP64 = 0, MIXED = 1, FP32 = 2 };
template <int KIND>
using Value = typename std::conditional<KIND == FP32, float, double>::type;

template <int DIM, int NC, int KIND>
__global__ void __launch_bounds__(kClusterThreads, 1)
    pcg_cluster(FaceOp<DIM, Value<KIND>> A, uint32_t n, uint32_t len, FastDiv dlen, IoT<Value<KIND>> P) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ TeamSmem ts;
  auto team = cluster_team<kClusterThreads>(&ts, len, dlen);
  cg_run<kClusterThreads, NC, (NC <= 2), true, true, KIND == MIXED>(
      A, n, len, P, team, reinterpret_cast<Value<KIND>*>(sm));
}

template <int DIM, int T, int NC, bool XS, bool HALO, int KIND>
__global__ void __launch_bounds__(T, 1)
    pcg_grid(FaceOp<DIM, Value<KIND>> A, uint32_t n, uint32_t len, GridWords w, IoT<Value<KIND>> P) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ TeamSmem ts;
  auto team = grid_team<T>(&ts, w);
  cg_run<T, NC, false, XS, HALO, KIND == MIXED>(A, n, len, P, team, reinterpret_cast<Value<KIND>*>(sm));
}

using ClusterNCs = std::integer_sequence<int, 1, 2, 3, 4, 6, 8>;
using SmallNCs = std::integer_sequence<int, 1, 2, 4>;
using LargeNCs = std::integer_sequence<int, 4, 8, 14>;

template <int DIM, int KIND>
cfdb_status run(cfdb_context* ctx, const OpView<Value<KIND>>& V, const Value<KIND>* invd,
                const IoT<Value<KIND>>& io) {
  const int64_t cells = (int64_t)V.nx * V.ny * V.nz;
  const int limit = cluster_limit((const void*)pcg_cluster<DIM, 8, KIND>, kClusterThreads);
  const Plan P = cg_plan(cells, (int64_t)V.nx * V.ny, ctx->num_sms, limit, sizeof(Value<KIND>));
  const uint32_t n = (uint32_t)cells;
  const FaceOp<DIM, Value<KIND>> A = face_op<DIM>(V, invd);
  GridWords w;
  cfdb_status st = prepare_words(ctx, P, &w);
  if (st != CFDB_OK) return st;
  CFDB_CUDA(ctx, cudaEventRecord(ctx->ev_k0, ctx->stream));
  cudaError_t e;
  if (P.team == 1) {
    e = with_nc(P.nc, ClusterNCs{}, [&](auto nc) {
      auto fn = pcg_cluster<DIM, decltype(nc)::value, KIND>;
      if (cluster_limit((const void*)fn, kClusterThreads) < P.blocks) return cudaErrorInvalidConfiguration;
      return launch_cluster(fn, P.blocks, P.blocks, kClusterThreads, P.smem, ctx->stream, A, n, P.len,
                            fast_div(P.len), io);
    });
  } else {
    auto go = [&](auto threads, auto nc) {
      constexpr int T = decltype(threads)::value, NC = decltype(nc)::value;
      const void* fn = P.halo ? (P.xs ? (const void*)pcg_grid<DIM, T, NC, true, true, KIND>
                                      : (const void*)pcg_grid<DIM, T, NC, false, true, KIND>)
                              : (P.xs ? (const void*)pcg_grid<DIM, T, NC, true, false, KIND>
                                      : (const void*)pcg_grid<DIM, T, NC, false, false, KIND>);
      cudaError_t q = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
      if (q != cudaSuccess) return q;
      auto a = A;
      uint32_t nn = n, len = P.len;
      auto o = io;
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

template <typename V>
IoT<V> io_of(cfdb_context* ctx, const V* b, V* x, V* pub, V* inv, const ResidentLimits& l) {
  IoT<V> io{};
  io.b = b;
  io.x = x;
  io.pub = pub;
  io.inv = inv;
  io.abs_tol = l.abs_tol;
  io.rel_tol = l.rel_tol;
  io.max_it = l.max_it;
  io.hist = l.hist;
  io.hist_cap = l.hist_cap;
  io.out = ctx->scalars;
  io.delta = l.delta;
  io.reps = ctx->scalars + l.reps_slot;
  return io;
}

}  // namespace

bool resident_pcg_fits(const cfdb_context* ctx, int nx, int ny, int nz, size_t word) {
  return cg_plan((int64_t)nx * ny * nz, (int64_t)nx * ny, ctx->num_sms, 0, word).team != 0;
}

cfdb_status resident_pcg(cfdb_context* ctx, const OpView<double>& A, int dim, const double* invd,
                         const double* b, double* x, double* pub, double* inv, const ResidentLimits& l) {
  const auto io = io_of<double>(ctx, b, x, pub, inv, l);
  if (l.delta > 0.0) return dim == 2 ? run<2, MIXED>(ctx, A, invd, io) : run<3, MIXED>(ctx, A, invd, io);
  return dim == 2 ? run<2, FP64>(ctx, A, invd, io) : run<3, FP64>(ctx, A, invd, io);
}

cfdb_status resident_pcg(cfdb_context* ctx, const OpView<float>& A, int dim, const float* invd,
                         const float* b, float* x, float* pub, float* inv, const ResidentLimits& l) {
  const auto io = io_of<float>(ctx, b, x, pub, inv, l);
  return dim == 2 ? run<2, FP32>(ctx, A, invd, io) : run<3, FP32>(ctx, A, invd, io);
}

}  // namespace cfdb
