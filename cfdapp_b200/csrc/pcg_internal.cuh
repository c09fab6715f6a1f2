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
// The on-chip FP64 Jacobi-PCG (resident_faces.cu): whether a system
// fits, and the solve (x in and out; `pub`, `inv`: vectors of `cells`,
// inv null where invd is given).  The
// outcome lands in the context's scalars.
bool resident_pcg_fits(const cfdb_context* ctx, const OpView<double>& A);
cfdb_status resident_pcg(cfdb_context* ctx, const OpView<double>& A, int dim, const double* invd,
                         const double* b, double* x, double* pub, double* inv,
                         double abs_tol, double rel_tol,
                         int64_t max_it, double* hist, int64_t hist_cap);
}
