// Internal entry points of the p' operator shared with the SIMPLE driver.
#pragma once

#include <cstdint>

#include "cfdb.h"
#include "poperator.cuh"

namespace cfdb {
struct LearnedSolver;
struct FineOperator;
cfdb_status poperator_bind_faces(cfdb_context* ctx, cfdb_poperator* op, const double* D, bool fp32);
// The operator as the learned preconditioner sees it, with its solver state
// (created on first use) and coefficient version.
void poperator_learned(cfdb_poperator* op, FineOperator* fo, LearnedSolver** solver,
                       uint64_t* version);
// The on-chip Jacobi-PCG (resident_faces.cu).
struct ResidentLimits {
  double abs_tol, rel_tol;
  int64_t max_it;
  double* hist;  // device, hist_cap entries
  int64_t hist_cap;
  double delta;   // > 0 (double vectors): mixed precision, residual replaced after this drop
  int reps_slot;  // context scalar that counts the replacements
};
// Whether a system (kernel-space extents, vectors of `word` bytes) fits.
bool resident_pcg_fits(const cfdb_context* ctx, int nx, int ny, int nz, size_t word);
// The solve, x in and out; pub, inv: vectors of the grid's cells (inv null
// where invd is given).  The outcome lands in the context's scalars.
cfdb_status resident_pcg(cfdb_context* ctx, const OpView<double>& A, int dim, const double* invd,
                         const double* b, double* x, double* pub, double* inv, const ResidentLimits& l);
cfdb_status resident_pcg(cfdb_context* ctx, const OpView<float>& A, int dim, const float* invd,
                         const float* b, float* x, float* pub, float* inv, const ResidentLimits& l);
}
