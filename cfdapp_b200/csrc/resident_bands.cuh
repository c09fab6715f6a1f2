// Launches of the on-chip stencil Krylov solves (resident_bands.cu), one
// dimension and method per translation unit: a process loads only the
// modules it runs.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

#include "resident_launch.cuh"
#include "stencil_solve.cuh"

namespace cfdb {
namespace res {

template <int DIM, bool PREC>
cudaError_t launch_bicgstab(cfdb_context* ctx, const BandOp<DIM>& A, const Plan& P, uint32_t n,
                            const GridWords& w, const Io& io);
template <int DIM>
int bicgstab_cluster_limit();
template <int DIM>
cudaError_t launch_cg(cfdb_context* ctx, const BandOp<DIM>& A, const Plan& P, uint32_t n,
                      const GridWords& w, const Io& io);
template <int DIM>
int cg_cluster_limit();

template <int DIM>
inline cudaError_t cooperative(const void* fn, const Plan& P, cudaStream_t st, BandOp<DIM> A, uint32_t n,
                        GridWords w, Io io) {
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
  if (e != cudaSuccess) return e;
  uint32_t len = P.len;
  void* args[] = {&A, &n, &len, &w, &io};
  return cudaLaunchCooperativeKernel(fn, dim3(P.blocks), dim3(P.threads), args, P.smem, st);
}

}  // namespace res
}  // namespace cfdb
