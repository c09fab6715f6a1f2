// The Jacobi-PCG of the p' operator with its vectors on chip (resident.cuh):
// the systems that fit one thread-block cluster, or the shared memory of the
// whole GPU.  FP64, mixed precision (FP32 directions) and FP32 (the inner
// solves of the refinement form).  A mixed solve (us per iteration, streaming
// kernel before): 128^2 3.8 (18.3), 64^3 10.6 (19.1), 96x80x64 14.5 (27.7),
// 128^3 34.3 (43.2); a refinement's FP32 iteration: 130x128 4.8 (12.0),
// 65x60x50 9.7 (24.3), 127x120x100 24.2 (61.9).
#include "resident_faces.cuh"

namespace cfdb {
namespace {

using namespace res;

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
  if (l.delta > 0.0) return dim == 2 ? pcg_on_chip<2, MIXED>(ctx, A, invd, io) : pcg_on_chip<3, MIXED>(ctx, A, invd, io);
  return dim == 2 ? pcg_on_chip<2, FP64>(ctx, A, invd, io) : pcg_on_chip<3, FP64>(ctx, A, invd, io);
}

cfdb_status resident_pcg(cfdb_context* ctx, const OpView<float>& A, int dim, const float* invd,
                         const float* b, float* x, float* pub, float* inv, const ResidentLimits& l) {
  const auto io = io_of<float>(ctx, b, x, pub, inv, l);
  return dim == 2 ? pcg_on_chip<2, FP32>(ctx, A, invd, io) : pcg_on_chip<3, FP32>(ctx, A, invd, io);
}

}  // namespace cfdb
