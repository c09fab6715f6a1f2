// Included by the resident_faces_*.cu that instantiate pcg_on_chip.
#pragma once

#include "resident_faces.cuh"

namespace cfdb {
namespace res {
namespace {

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

}  // namespace

template <int DIM, int KIND>
cfdb_status pcg_on_chip(cfdb_context* ctx, const OpView<Value<KIND>>& V, const Value<KIND>* invd,
                        const IoT<Value<KIND>>& io) {
  const int64_t cells = (int64_t)V.nx * V.ny * V.nz;
  const int limit = cells <= cluster_cells(DIM)
                        ? cluster_limit((const void*)pcg_cluster<DIM, 8, KIND>, kClusterThreads)
                        : 0;
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
      const void* fn = P.halo ? (const void*)pcg_grid<DIM, T, NC, true, true, KIND>
                              : (const void*)pcg_grid<DIM, T, NC, true, false, KIND>;
      if constexpr (T == kGridThreadsLarge) {  // a small block's x always fits (cg_plan)
        if (!P.xs && P.halo) fn = (const void*)pcg_grid<DIM, T, NC, false, true, KIND>;
        // alone, p, r and x leave the block's memory only at the most cells a thread
        if constexpr ((size_t)3 * NC * T * sizeof(Value<KIND>) > kSmemMax)
          if (!P.xs && !P.halo) fn = (const void*)pcg_grid<DIM, T, NC, false, false, KIND>;
      }
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

}  // namespace res
}  // namespace cfdb
