// The stencil Krylov solves (BiCGSTAB, CG, optional Jacobi) with their
// vectors on chip (resident.cuh), for the systems that fit.
#include "resident_bands.cuh"

namespace cfdb {
namespace {

using namespace res;

template <int DIM>
cfdb_status run(cfdb_context* ctx, const StencilMatrix& M, int krylov, const Io& io, bool* taken) {
  *taken = false;
  int limit = 0;  // asked for where a cluster may take the system
  if (krylov == 1 && M.n <= kBicgClusterCells) limit = bicgstab_cluster_limit<DIM>();
  if (krylov != 1 && M.n <= cluster_cells(DIM)) limit = cg_cluster_limit<DIM>();
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
