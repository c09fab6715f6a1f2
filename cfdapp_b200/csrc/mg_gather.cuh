// V-cycle and FCG passes for the levels the quad kernels do not take (rows
// that are not a multiple of 4 or shorter than a tile, and levels too small
// for a march to pay): one cell per thread, every operand a plain load.
// Included by mg.cu inside its anonymous namespace.
//
// A pass over such a level is bound by the latency of its loads, which L1
// and L2 serve, not by their number: a thread issues all its loads at once --
// a neighbour outside the domain is read at the cell itself and counted 0, so
// no load waits behind a branch -- with 32-bit indices and divisions by
// multiplication.  Marching blocks along z through shared-memory planes
// instead chains a barrier and a load per plane.  FCG iteration (us, one-cell
// marching kernels before): 100x75x61 102 (127), 80x48x48 82 (92), 1001x900
// 115 (148), 2047x2045 286 (373), 255x253x251 1288 (1709).
#pragma once

struct GLevel {
  LV L;
  res::FastDiv dx, dy;
  uint32_t n;
};

GLevel glevel(const MgLevel& M) {
  GLevel G;
  G.L = lv(M);
  G.dx = res::fast_div(M.n[0]);
  G.dy = res::fast_div(M.n[1]);
  G.n = (uint32_t)M.cells;
  return G;
}

// Blocks of a pass over n cells: one cell a thread up to the widest reduction.
int gather_blocks(int64_t n) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, kMaxBlocks));
}

using res::gather_cells;

// Couplings of a cell (coef() with 32-bit indices).
template <int DIM>
__device__ __forceinline__ C7 gather_coef(const LV& L, uint32_t c, int j, int k) {
  C7 o;
  const uint32_t row = j + L.ny * k;
  o.xl = L.fx[c + row];
  o.xh = L.fx[c + row + 1];
  o.yl = DIM == 3 ? L.fy[c + L.nx * k] : 0.f;
  o.yh = DIM == 3 ? L.fy[c + L.nx * k + L.nx] : 0.f;
  o.zl = L.fz[c];
  o.zh = L.fz[c + L.nx * L.ny];
  o.d = ((o.xl + o.xh) + (o.yl + o.yh)) + (o.zl + o.zh);
  return o;
}

// (A v)(c); val(q, di, dj, dk) is v at cell q = c + offset.
template <int DIM, class Val>
__device__ __forceinline__ float gather_lap(const LV& L, uint32_t c, int i, int j, int k, Val val) {
  const int plane = L.nx * L.ny;
  auto at = [&](bool in, int off, int di, int dj, int dk) {
    const float v = val(in ? c + off : c, in ? di : 0, in ? dj : 0, in ? dk : 0);
    return in ? v : 0.f;
  };
  const float v = val(c, 0, 0, 0);
  const float w = at(i > 0, -1, -1, 0, 0), e = at(i + 1 < L.nx, 1, 1, 0, 0);
  const float s = DIM == 3 ? at(j > 0, -L.nx, 0, -1, 0) : 0.f;
  const float n = DIM == 3 ? at(j + 1 < L.ny, L.nx, 0, 1, 0) : 0.f;
  const float b = at(k > 0, -plane, 0, 0, -1), t = at(k + 1 < L.nz, plane, 0, 0, 1);
  return apply7(gather_coef<DIM>(L, c, j, k), v, w, e, s, n, b, t);
}

// sum_o K[o] u(c + o), taps in (dz, dy, dx) order.
template <int DIM, class U>
__device__ __forceinline__ float gather_conv(const LV& L, const Kern& K, uint32_t c, int i, int j, int k, U u) {
  float sum = 0.f;
#pragma unroll
  for (int dk = -1; dk <= 1; ++dk) {
    const bool zin = k + dk >= 0 && k + dk < L.nz;
#pragma unroll
    for (int dj = (DIM == 2 ? 0 : -1); dj <= (DIM == 2 ? 0 : 1); ++dj) {
      const bool yin = zin && (DIM == 2 || (j + dj >= 0 && j + dj < L.ny));
      const uint32_t q = c + dk * L.nx * L.ny + dj * L.nx;
#pragma unroll
      for (int di = -1; di <= 1; ++di) {
        const bool in = yin && i + di >= 0 && i + di < L.nx;
        const float v = u(in ? q + di : c);
        sum += K.w[(dk + 1) * 9 + (dj + 1) * 3 + (di + 1)] * (in ? v : 0.f);
      }
    }
  }
  return sum;
}

__device__ __forceinline__ int gather_parent(const LV& C, int i, int j, int k) {
  return (i >> 1) + C.nx * ((j >> 1) + C.ny * (k >> 1));
}

// x = D^-1/2 (W * (D^-1/2 r)), r[skip] read as 0
template <int DIM>
__global__ void __launch_bounds__(256) k_first_g(GLevel G, Kern K, const float* __restrict__ r,
                                                 float* __restrict__ x, uint32_t skip) {
  pdl_enter();
  const LV& L = G.L;
  gather_cells(G.n, L.nx, L.ny, G.dx, G.dy, [&](uint32_t c, int i, int j, int k) {
    const float s = gather_conv<DIM>(L, K, c, i, j, k, [&](uint32_t q) {
      const float v = r[q] * L.isq[q];
      return q == skip ? 0.f : v;
    });
    x[c] = L.isq[c] * s;
  });
}

// rc = sum of the children's (r - A x)
template <int DIM>
__global__ void __launch_bounds__(256) k_restrict_g(GLevel G, GLevel C, const float* __restrict__ x,
                                                    const float* __restrict__ r,
                                                    float* __restrict__ rc, uint32_t skip) {
  pdl_enter();
  const LV& L = G.L;
  gather_cells(C.n, C.L.nx, C.L.ny, C.dx, C.dy, [&](uint32_t qc, int ci, int cj, int ck) {
    float sum = 0.f;
#pragma unroll
    for (int u = 0; u < 2; ++u)
#pragma unroll
      for (int v = 0; v < (DIM == 3 ? 2 : 1); ++v)
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          const int i = 2 * ci + t, j = DIM == 3 ? 2 * cj + v : 0, k = 2 * ck + u;
          if (i < L.nx && j < L.ny && k < L.nz) {
            const uint32_t c = i + L.nx * (j + L.ny * k);
            const float ax = gather_lap<DIM>(L, c, i, j, k, [&](uint32_t q, int, int, int) { return x[q]; });
            sum += (c == skip ? 0.f : r[c]) - ax;
          }
        }
    rc[qc] = sum;
  });
}

// u = D^-1/2 (r - A x) (PRO: x + cw P ec in place of x)
template <int DIM, bool PRO>
__global__ void __launch_bounds__(256) k_resid_g(GLevel G, LV C, const float* __restrict__ x,
                                                 const float* __restrict__ ec, float cw,
                                                 const float* __restrict__ r, float* __restrict__ u,
                                                 uint32_t skip) {
  pdl_enter();
  const LV& L = G.L;
  gather_cells(G.n, L.nx, L.ny, G.dx, G.dy, [&](uint32_t c, int i, int j, int k) {
    const float ax = gather_lap<DIM>(L, c, i, j, k, [&](uint32_t q, int di, int dj, int dk) {
      float v = x[q];
      if (PRO) v += cw * ec[gather_parent(C, i + di, j + dj, k + dk)];
      return v;
    });
    u[c] = L.isq[c] * ((c == skip ? 0.f : r[c]) - ax);
  });
}

// x += [cw P ec] + D^-1/2 (W * u); pin >= 0: x[pin] = r[pin]; HOOK: z.q
template <int DIM, bool HOOK>
__global__ void __launch_bounds__(256) k_smooth_g(GLevel G, LV C, Kern K, const float* __restrict__ u,
                                                  const float* __restrict__ ec, float cw,
                                                  float* __restrict__ x, uint32_t pin,
                                                  const float* __restrict__ r, Hook hk) {
  pdl_enter();
  const LV& L = G.L;
  double acc[1] = {0.0};
  gather_cells(G.n, L.nx, L.ny, G.dx, G.dy, [&](uint32_t c, int i, int j, int k) {
    const float s = gather_conv<DIM>(L, K, c, i, j, k, [&](uint32_t q) { return u[q]; });
    float v = L.isq[c] * s + x[c];
    if (ec) v += cw * ec[gather_parent(C, i, j, k)];
    if (c == pin) v = r[c];
    x[c] = v;
    if (HOOK) acc[0] += (double)v * hk.q[c];
  });
  if (HOOK) {
    reduce_last<1>(acc, hk.partials, &hk.S->ticket, [&](const double* tot) {
      FcgState* S = hk.S;
      if (S->it == 0) return;  // the first direction is z itself
      const double beta = tot[0] / S->pq;
      if (!isfinite(beta)) {
        stop_loop(S, hk.h, kLearnedStagnated);
        return;
      }
      S->beta = beta;
    });
  }
}

// p = z - beta p_old (p = z on the first iteration), q = A p; p.q, p.r
template <int DIM>
__global__ void __launch_bounds__(256) k_fcg_dir_g(res::FaceOp<DIM> A, uint32_t n, FcgState* S,
                                                   const float* __restrict__ z, double* P0, double* P1,
                                                   double* __restrict__ q, const double* __restrict__ r,
                                                   double* partials, Loop h) {
  pdl_enter();
  if (S->done) return;
  const long long it = S->it;
  const bool first = (it == 0);
  const double beta = first ? 0.0 : S->beta;
  double* __restrict__ pn = (it & 1) ? P1 : P0;
  const double* __restrict__ po = (it & 1) ? P0 : P1;
  auto val = [&](uint32_t c) {
    const double v = (double)z[c];
    return first ? v : fma(-beta, po[c], v);
  };
  double acc[2] = {0.0, 0.0};
  const int sz = (int)A.sz;
  gather_cells(n, A.nx, A.ny, A.dx, A.dy, [&](uint32_t c, int i, int j, int k) {
    const res::Cf<double> f = A.load(c, i, j, k);
    // (couplings across the domain's edge are 0: any value inside will do)
    const double v = val(c);
    const double w = val(i > 0 ? c - 1 : c), e = val(i + 1 < A.nx ? c + 1 : c);
    const double s = DIM == 3 ? val(j > 0 ? c - A.nx : c) : 0.0;
    const double nn = DIM == 3 ? val(j + 1 < A.ny ? c + A.nx : c) : 0.0;
    const double b = val(k > 0 ? c - sz : c), t = val(k + 1 < A.nz ? c + sz : c);
    const double aq = A.mul(f, v, w, e, s, nn, b, t);
    pn[c] = v;
    q[c] = aq;
    acc[0] += v * aq;
    acc[1] += v * r[c];
  });
  reduce_last<2>(acc, partials, &S->ticket, [&](const double* tot) {
    const double pq = tot[0], pr = tot[1];
    const double alpha = pr / pq;
    if (!isfinite(pq) || !(pq > 0.0) || !isfinite(alpha)) {
      stop_loop(S, h, kLearnedStagnated);
      return;
    }
    S->pq = pq;
    S->pr = pr;
    S->alpha = alpha;
  });
}
