// V-cycle levels and whole FCG solves on one thread-block cluster (included
// by mg.cu inside its anonymous namespace).
//
// A pass over a level of a few thousand cells is all latency: as a kernel of
// its own it takes 3.5-4 us, and inside one kernel with its vectors in L2 and
// a cluster barrier between passes still 2 us (a trip to L2 for the loads and
// one for the stores before the barrier).  Here the vectors of the small
// levels live in the shared memory of a cluster of 16 blocks of 512 threads
// (with 1024 the barriers and sums cost more than the passes gain: an FCG
// iteration of 24^2 14.3 against 10.4 us, 129^2 29.5 / 26.6, 24^3 36.9 / 28.9).
// Every block owns a run of planes of each level (z in kernel space), aligned
// so that a coarse plane's children belong to its owner; each vector that a
// stencil reads keeps one halo plane per side, which the neighbours push into
// it through distributed shared memory as they compute; a hardware cluster
// barrier ends each pass.  Couplings and scales come through L1.  The
// coarsest levels run in the first block (coarse_cycle).  What bounds it now
// is instruction issue and the chain of passes on 16 SMs.
//
//   k_tail         the levels below the grid kernels' in one launch
//   k_fcg_cluster  the whole FCG loop of a small system: one launch a solve
#pragma once

constexpr int kClusterT = 512;
constexpr int kMaxTail = 6;

using ClusterT = res::ClusterTeam<kClusterT>;

struct TailLevel {
  LV L;
  res::FastDiv dx, dy;
  int planes;         // planes per block (the last blocks may have fewer)
  int ox, ou, orr;    // shared-memory offsets (floats) of x, u (windows), r
  float cw;
  Kern K;
};

struct TailPlan {
  int count;  // levels run by the whole cluster
  int nu;
  int coarse;  // offset (floats) of the block-resident levels' memory
  int oe;      // offset of the first block-resident level's x window
  int ep;      // planes of that level per block
  int op, or64, oq, ox64;  // FCG: offsets (floats) of p (window), r, q, x; ox64 < 0: x in memory
  TailLevel lv[kMaxTail];
  LV C;  // the first block-resident level
  res::FastDiv cdx, cdy;
  const float* r_glob;  // k_tail: the first level's right-hand side and result
  float* x_glob;
};

// The plans' copies lead the dynamic shared memory.
constexpr int kPlanWords = plan_words<TailPlan>() + plan_words<CoarsePlan>();

// One block's share of a level.
struct Share {
  int z0, np;      // first plane and number of planes
  bool lo, hi;     // neighbours before and after
  int plane;
};
__device__ __forceinline__ Share share_of(const LV& L, int planes, int rank) {
  Share s;
  s.z0 = min(L.nz, planes * rank);
  s.np = min(planes, L.nz - s.z0);
  s.lo = s.np > 0 && s.z0 > 0;
  s.hi = s.np > 0 && s.z0 + s.np < L.nz;
  s.plane = L.nx * L.ny;
  return s;
}

template <typename E>
__device__ __forceinline__ void put_remote(const E* at, int rank, E v) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(at);
  uint32_t ra;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(ra), "f"(v) : "memory");
}
__device__ __forceinline__ float get_remote(const float* at, int rank) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(at);
  uint32_t ra;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(ra) : "memory");
  return v;
}

// f(t, c, i, j, kl): own cell t (global c) at (i, j) of own plane kl.
template <class F>
__device__ __forceinline__ void own_cells(const LV& L, res::FastDiv dx, res::FastDiv dy, const Share& S, F f) {
  const int n = S.np * S.plane;
  for (int t = threadIdx.x; t < n; t += kClusterT) {
    const uint32_t row = dx.div((uint32_t)t);
    const uint32_t kl = dy.div(row);
    f(t, S.z0 * S.plane + t, (int)(t - row * (uint32_t)L.nx), (int)(row - kl * (uint32_t)L.ny), (int)kl);
  }
}

// Stores v at cell (own index t, plane kl) of a window (one plane before the
// first own one) and in the neighbours' halos of it.
__device__ __forceinline__ void put(float* win, const Share& S, int planes, int rank, int t, int kl, float v) {
  win[S.plane + t] = v;
  if (kl == 0 && S.lo) put_remote(win + (planes + 1) * S.plane + t, rank - 1, v);
  if (kl == S.np - 1 && S.hi) put_remote(win + t - (S.np - 1) * S.plane, rank + 1, v);
}

// Couplings of a cell (coef() with 32-bit indices, k the plane in the level).
template <int DIM>
__device__ __forceinline__ C7 coef32(const LV& L, int c, int j, int k) {
  C7 o;
  const int row = j + L.ny * k;
  o.xl = __ldg(L.fx + c + row);
  o.xh = __ldg(L.fx + c + row + 1);
  if (DIM == 3) {
    o.yl = __ldg(L.fy + c + L.nx * k);
    o.yh = __ldg(L.fy + c + L.nx * k + L.nx);
  } else {
    o.yl = o.yh = 0.f;
  }
  o.zl = __ldg(L.fz + c);
  o.zh = __ldg(L.fz + c + L.nx * L.ny);
  o.d = ((o.xl + o.xh) + (o.yl + o.yh)) + (o.zl + o.zh);
  return o;
}

// (A v)(c): val(d, di, dj, dk) is v at the cell's offset; places outside the
// domain in x and y are read (inside the window's padding) and count 0, the
// halo planes outside it in z hold zeros.
template <int DIM, class Val>
__device__ __forceinline__ float lap32(const LV& L, int c, int i, int j, int k, Val val) {
  const int plane = L.nx * L.ny;
  const float v = val(0, 0, 0, 0);
  const float w0 = val(-1, -1, 0, 0), e0 = val(1, 1, 0, 0);
  const float w = i > 0 ? w0 : 0.f, e = i + 1 < L.nx ? e0 : 0.f;
  float s = 0.f, n = 0.f;
  if (DIM == 3) {
    const float s0 = val(-L.nx, 0, -1, 0), n0 = val(L.nx, 0, 1, 0);
    s = j > 0 ? s0 : 0.f;
    n = j + 1 < L.ny ? n0 : 0.f;
  }
  const float b = k > 0 ? val(-plane, 0, 0, -1) : 0.f, t = k + 1 < L.nz ? val(plane, 0, 0, 1) : 0.f;
  return apply7(coef32<DIM>(L, c, j, k), v, w, e, s, n, b, t);
}

// sum_o K[o] u(c + o), taps in (dz, dy, dx) order, `u` at the cell in a window.
template <int DIM>
__device__ __forceinline__ float conv32(const LV& L, const Kern& K, int i, int j, const float* u) {
  const bool xl = i > 0, xh = i + 1 < L.nx;
  float sum = 0.f;
#pragma unroll
  for (int dk = -1; dk <= 1; ++dk)
#pragma unroll
    for (int dj = (DIM == 2 ? 0 : -1); dj <= (DIM == 2 ? 0 : 1); ++dj) {
      const float* row = u + dk * L.nx * L.ny + dj * L.nx;
      const bool yin = DIM == 2 || dj == 0 || (dj < 0 ? j > 0 : j + 1 < L.ny);
      const float a = row[-1], b = row[0], c = row[1];
      const float* w = K.w + (dk + 1) * 9 + (dj + 1) * 3;
      sum += w[0] * (xl && yin ? a : 0.f);
      sum += w[1] * (yin ? b : 0.f);
      sum += w[2] * (xh && yin ? c : 0.f);
    }
  return sum;
}

// z = M r over the plan's levels.  On entry level 0's u = D^-1/2 r window is
// in place (halos included, a barrier passed); on exit its x window holds z
// (the barrier after the last pass is the caller's).  r0(t): level 0's r;
// pin: the own index of the pinned cell, whose z is rpin, or -1; done(t, z)
// runs per own cell.
template <int DIM, class R0, class Done>
__device__ __forceinline__ void tail_cycle(const TailPlan& P, const CoarsePlan& Q, ClusterT& T,
                                           float* sm, R0 r0, int pin, float rpin, Done done) {
  const int rank = T.rank_;
  auto scale = [&](const TailLevel& V, int c) { return __ldg(V.L.isq + c); };
  auto rhs = [&](int l, const TailLevel& V, int t) { return l == 0 ? r0(t) : sm[V.orr + t]; };
  // u = D^-1/2 (r - A x), pushed
  auto residual = [&](int l, const TailLevel& V, const Share& S) {
    const float* X = sm + V.ox + S.plane;
    own_cells(V.L, V.dx, V.dy, S, [&](int t, int c, int i, int j, int kl) {
      const float* x = X + t;
      const float ax = lap32<DIM>(V.L, c, i, j, S.z0 + kl, [&](int d, int, int, int) { return x[d]; });
      put(sm + V.ou, S, V.planes, rank, t, kl, scale(V, c) * (rhs(l, V, t) - ax));
    });
  };
  // x += D^-1/2 (W * u), pushed
  auto smooth = [&](const TailLevel& V, const Share& S) {
    const float* U = sm + V.ou + S.plane;
    const float* X = sm + V.ox + S.plane;
    own_cells(V.L, V.dx, V.dy, S, [&](int t, int c, int i, int j, int kl) {
      put(sm + V.ox, S, V.planes, rank, t, kl, X[t] + scale(V, c) * conv32<DIM>(V.L, V.K, i, j, U + t));
    });
  };
  for (int l = 0; l < P.count; ++l) {
    const TailLevel V = P.lv[l];
    const Share S = share_of(V.L, V.planes, rank);
    const float* U = sm + V.ou + S.plane;
    own_cells(V.L, V.dx, V.dy, S, [&](int t, int c, int i, int j, int kl) {
      put(sm + V.ox, S, V.planes, rank, t, kl, scale(V, c) * conv32<DIM>(V.L, V.K, i, j, U + t));
    });
    T.sync();
    for (int s = 1; s < P.nu; ++s) {
      residual(l, V, S);
      T.sync();
      smooth(V, S);
      T.sync();
    }
    // the residual into u's own cells, then the restriction: children are own cells
    float* W = sm + V.ou + S.plane;
    const float* X = sm + V.ox + S.plane;
    own_cells(V.L, V.dx, V.dy, S, [&](int t, int c, int i, int j, int kl) {
      const float* x = X + t;
      W[t] = rhs(l, V, t) - lap32<DIM>(V.L, c, i, j, S.z0 + kl, [&](int d, int, int, int) { return x[d]; });
    });
    __syncthreads();
    const bool more = l + 1 < P.count;
    const LV& C = more ? P.lv[l + 1].L : P.C;
    const Share SC = share_of(C, more ? P.lv[l + 1].planes : P.ep, rank);
    const res::FastDiv cdx = more ? P.lv[l + 1].dx : P.cdx, cdy = more ? P.lv[l + 1].dy : P.cdy;
    own_cells(C, cdx, cdy, SC, [&](int t, int c, int ci, int cj, int ck) {
      float sum = 0.f;
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < (DIM == 3 ? 2 : 1); ++v)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int i = 2 * ci + q, j = DIM == 3 ? 2 * cj + v : 0, k = 2 * ck + u;
            if (i < V.L.nx && j < V.L.ny && k < S.np) sum += W[i + V.L.nx * (j + V.L.ny * k)];
          }
      if (more) {
        const TailLevel& N = P.lv[l + 1];
        sm[N.orr + t] = sum;
        put(sm + N.ou, SC, N.planes, rank, t, ck, scale(N, c) * sum);
      } else {
        put_remote(sm + P.coarse + Q.lv[0].off[5] + c, 0, sum);
      }
    });
    T.sync();
  }
  // the block-resident levels, then every block fetches its planes of their x
  float* cs = sm + P.coarse;
  if (rank == 0) {
    cp_wait<0>();
    __syncthreads();
    coarse_cycle<DIM>(Q, cs);
  }
  T.sync();
  {
    const Share S = share_of(P.C, P.ep, rank);
    const int first = S.lo ? -1 : 0, last = S.np + (S.hi ? 1 : 0);
    const int px = P.C.nx + 2, pz = DIM == 3 ? px * (P.C.ny + 2) : px;
    float* E = sm + P.oe + S.plane;
    for (int t = first * S.plane + (int)threadIdx.x; t < last * S.plane; t += kClusterT) {
      const uint32_t c = (uint32_t)(S.z0 * S.plane + t);
      const uint32_t row = P.cdx.div(c), k = P.cdy.div(row);
      const int i = (int)(c - row * (uint32_t)P.C.nx), j = (int)(row - k * (uint32_t)P.C.ny);
      E[t] = get_remote(cs + Q.lv[0].off[4] + (i + 1) + (DIM == 3 ? px * (j + 1) : 0) + pz * ((int)k + 1), 0);
    }
    __syncthreads();
  }
  for (int l = P.count - 1; l >= 0; --l) {
    const TailLevel& V = P.lv[l];
    const Share S = share_of(V.L, V.planes, rank);
    const bool more = l + 1 < P.count;
    const LV& C = more ? P.lv[l + 1].L : P.C;
    const int cplane = C.nx * C.ny;
    const float* E = sm + (more ? P.lv[l + 1].ox : P.oe) + cplane;
    // (the own planes start at twice the coarse ones)
    auto ec = [&](int i, int j, int kl) {
      return E[(i >> 1) + C.nx * ((j >> 1) + C.ny * (kl >> 1))];
    };
    const float* X = sm + V.ox + S.plane;
    const float* U = sm + V.ou + S.plane;
    for (int s = 0; s < P.nu; ++s) {
      const bool last = l == 0 && s == P.nu - 1;
      if (s == 0) {
        own_cells(V.L, V.dx, V.dy, S, [&](int t, int c, int i, int j, int kl) {
          const float* x = X + t;
          const float ax = lap32<DIM>(V.L, c, i, j, S.z0 + kl, [&](int d, int di, int dj, int dk) {
            return x[d] + V.cw * ec(i + di, j + dj, kl + dk);
          });
          put(sm + V.ou, S, V.planes, rank, t, kl, scale(V, c) * (rhs(l, V, t) - ax));
        });
      } else {
        residual(l, V, S);
      }
      T.sync();
      own_cells(V.L, V.dx, V.dy, S, [&](int t, int c, int i, int j, int kl) {
        float v = scale(V, c) * conv32<DIM>(V.L, V.K, i, j, U + t) + X[t];
        if (s == 0) v += V.cw * ec(i, j, kl);
        if (last && t == pin) v = rpin;
        put(sm + V.ox, S, V.planes, rank, t, kl, v);
        if (last) done(t, v);
      });
      if (!last) T.sync();
    }
  }
}

// Zeroes the cluster kernel's shared memory (halos outside the domain stay
// zero) and, in the first block, brings in the block-resident levels.
template <int DIM>
__device__ __forceinline__ void tail_setup(const TailPlan& P, const CoarsePlan& Q, float* sm,
                                           int words, int rank) {
  // (every offset is a multiple of four floats)
  for (int q = kPlanWords + 4 * threadIdx.x; q < words; q += 4 * kClusterT)
    *reinterpret_cast<float4*>(sm + q) = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  if (rank == 0) {
    coarse_fetch_levels<DIM>(Q, sm + P.coarse);  // lands by the first coarse cycle
    cp_commit();
  }
}

__device__ __forceinline__ ClusterT own_team(res::TeamSmem* ts) {
  return res::cluster_team<kClusterT>(ts, 1, res::FastDiv{});
}

template <int DIM>
__global__ void __launch_bounds__(kClusterT, 1)
    k_tail(const __grid_constant__ TailPlan P0, const __grid_constant__ CoarsePlan Q0, int words) {
  extern __shared__ float4 smem4[];
  __shared__ res::TeamSmem ts;
  float* sm = reinterpret_cast<float*>(smem4);
  const TailPlan& P = to_shared(P0, sm);
  const CoarsePlan& Q = to_shared(Q0, sm + plan_words<TailPlan>());
  ClusterT T = own_team(&ts);
  tail_setup<DIM>(P, Q, sm, words, T.rank_);
  pdl_enter();
  const TailLevel& V = P.lv[0];
  const Share S = share_of(V.L, V.planes, T.rank_);
  own_cells(V.L, V.dx, V.dy, S, [&](int t, int c, int, int, int) { sm[V.orr + t] = __ldcg(P.r_glob + c); });
  // u with its halos, straight from the right-hand side
  const int first = S.lo ? -S.plane : 0, last = (S.np + (S.hi ? 1 : 0)) * S.plane;
  for (int t = first + (int)threadIdx.x; t < last; t += kClusterT) {
    const int c = S.z0 * S.plane + t;
    sm[V.ou + S.plane + t] = __ldg(V.L.isq + c) * __ldcg(P.r_glob + c);
  }
  T.sync();
  tail_cycle<DIM>(P, Q, T, sm, [&](int t) { return sm[V.orr + t]; }, -1, 0.f,
                  [&](int t, float z) { P.x_glob[S.z0 * S.plane + t] = z; });
  T.sync();  // no block leaves while another may still write into it
}

struct FcgArgs {
  OpView<double> A;
  FcgState* S;
  double* hist;
  int64_t hcap;
  int pin;  // the pinned cell or -1
};

// A whole FCG(1) solve of a small system: k_fcg_init, the V-cycle,
// direction pass and k_fcg_update of the graph form, with its stopping tests.
// p keeps halo planes that its readers update themselves from the pushed z.
template <int DIM>
__global__ void __launch_bounds__(kClusterT, 1)
    k_fcg_cluster(const __grid_constant__ FcgArgs F, const __grid_constant__ TailPlan P0,
                  const __grid_constant__ CoarsePlan Q0, int words) {
  extern __shared__ float4 smem4[];
  __shared__ res::TeamSmem ts;
  float* sm = reinterpret_cast<float*>(smem4);
  const TailPlan& P = to_shared(P0, sm);
  const CoarsePlan& Q = to_shared(Q0, sm + plan_words<TailPlan>());
  ClusterT T = own_team(&ts);
  tail_setup<DIM>(P, Q, sm, words, T.rank_);
  T.enter();  // and every block's memory is ready for its neighbours' values
  FcgState* S = F.S;
  const bool leader = T.rank_ == 0 && threadIdx.x == 0;
  const TailLevel& V = P.lv[0];
  const Share H = share_of(V.L, V.planes, T.rank_);
  const res::FaceOp<DIM> A = res::face_op<DIM>(F.A, (const double*)nullptr);
  const double* __restrict__ b = S->b;
  double* x = S->x;
  const double abs_tol = S->abs_tol, rel_tol = S->rel_tol;
  const long long max_it = S->max_it, window = S->window;
  double* p = reinterpret_cast<double*>(sm + P.op) + H.plane;
  double* r = reinterpret_cast<double*>(sm + P.or64);
  double* q = reinterpret_cast<double*>(sm + P.oq);
  double* xs = P.ox64 >= 0 ? reinterpret_cast<double*>(sm + P.ox64) : nullptr;
  const int base = H.z0 * H.plane;
  const int pin = F.pin >= base && F.pin < base + H.np * H.plane ? F.pin - base : -1;
  // u = D^-1/2 float(r) (0 at the pinned cell), pushed
  auto push_u = [&](int t, int c, int kl, double rn) {
    put(sm + V.ou, H, V.planes, T.rank_, t, kl, t == pin ? 0.f : __ldg(V.L.isq + c) * (float)rn);
  };
  auto stop = [&](int status, long long it, double res) {
    cp_wait<0>();  // no copy of the coarse levels is in flight when the block leaves
    if (leader) {
      S->it = it;
      S->res = res;
      S->status = status;
      S->done = 1;
    }
    if (xs && it > 0)
      for (int t = threadIdx.x; t < H.np * H.plane; t += kClusterT) x[base + t] = xs[t];
  };
  // ---- r = b - A x
  double one[1] = {0.0};
  own_cells(V.L, V.dx, V.dy, H, [&](int t, int c, int i, int j, int kl) {
    const double rn = __ldg(b + c) - res::apply_global(A, A.load(c, i, j, H.z0 + kl), c, x);
    r[t] = rn;
    if (xs) xs[t] = __ldcg(x + c);
    push_u(t, c, kl, rn);
    one[0] += rn * rn;
  });
  T.reduce(one);
  const double b0 = sqrt(one[0]);
  if (leader) {
    S->b0 = b0;
    if (F.hcap > 0) F.hist[0] = b0;
  }
  if (!isfinite(b0)) return stop(CFDB_SOLVER_NONFINITE_RESIDUAL, 0, b0);
  if (b0 == 0.0 || b0 <= abs_tol || 1.0 <= rel_tol) return stop(CFDB_SOLVER_CONVERGED, 0, b0);
  double best = b0, res = b0, pq = 1.0;
  long long best_it = 0;
  const int first = H.lo ? -H.plane : 0, last = (H.np + (H.hi ? 1 : 0)) * H.plane;
  for (long long it = 0;; ++it) {
    // ---- z = M r and z.q of the previous direction
    double zq[1] = {0.0};
    tail_cycle<DIM>(P, Q, T, sm, [&](int t) { return t == pin ? 0.f : (float)r[t]; }, pin,
                    pin >= 0 ? (float)r[pin] : 0.f, [&](int t, float z) {
                      if (it > 0) zq[0] += (double)z * q[t];
                    });
    T.reduce(zq);
    double beta = 0.0;
    if (it > 0) {
      beta = zq[0] / pq;
      if (!isfinite(beta)) return stop(kLearnedStagnated, it, res);
    }
    // ---- p = z - beta p (halo planes too), q = A p; p.q, p.r
    const float* z = sm + V.ox + H.plane;
    for (int t = first + (int)threadIdx.x; t < last; t += kClusterT)
      p[t] = it == 0 ? (double)z[t] : fma(-beta, p[t], (double)z[t]);
    __syncthreads();
    double pr[2] = {0.0, 0.0};
    own_cells(V.L, V.dx, V.dy, H, [&](int t, int c, int i, int j, int kl) {
      const double* v = p + t;
      const double aq = A.mul(A.load(c, i, j, H.z0 + kl), v[0], v[-1], v[1], DIM == 3 ? v[-A.nx] : 0.0,
                              DIM == 3 ? v[A.nx] : 0.0, v[-H.plane], v[H.plane]);
      q[t] = aq;
      pr[0] += v[0] * aq;
      pr[1] += v[0] * r[t];
    });
    T.reduce(pr);
    pq = pr[0];
    const double alpha = pr[1] / pq;
    if (!isfinite(pq) || !(pq > 0.0) || !isfinite(alpha)) return stop(kLearnedStagnated, it, res);
    // ---- x += alpha p, r -= alpha q
    double rr[1] = {0.0};
    own_cells(V.L, V.dx, V.dy, H, [&](int t, int c, int, int, int kl) {
      if (xs) xs[t] = fma(alpha, p[t], xs[t]);
      else x[c] = fma(alpha, p[t], x[c]);
      const double rn = fma(-alpha, q[t], r[t]);
      r[t] = rn;
      push_u(t, c, kl, rn);
      rr[0] += rn * rn;
    });
    T.reduce(rr);
    res = sqrt(rr[0]);
    const long long k = it + 1;
    if (leader && k < F.hcap) F.hist[k] = res;
    if (!isfinite(res)) return stop(CFDB_SOLVER_NONFINITE_RESIDUAL, k, res);
    if (res <= abs_tol || (b0 > 0.0 && res / b0 <= rel_tol)) return stop(CFDB_SOLVER_CONVERGED, k, res);
    if (res < best) {
      best = res;
      best_it = k;
    } else if (k - best_it >= window) {
      return stop(kLearnedStagnated, k, res);
    }
    if (k >= max_it) return stop(CFDB_SOLVER_MAX_ITERATIONS, k, res);
  }
}

// --------------------------------------------------------------- host side

// Layout of the levels [from, ...) in the cluster: levels of more than
// `block_cells` cells are spread over it.  words = 0 when they do not fit.
struct ClusterLayout {
  TailPlan P;
  CoarsePlan Q;
  int words = 0;
};

// Cells of the largest level left to the first block alone.  2D: 1600, about
// a cell and a half per thread; 3D: kCoarseCells, since splitting a level
// needs planes (16^3 gives every block one, 8^3 only half of them).
int64_t block_cells(int dim) { return dim == 2 ? 1600 : kCoarseCells; }

ClusterLayout cluster_layout(const MgHierarchy& H, const MgWeights& W, int from, bool fcg,
                             const float* r_glob, float* x_glob) {
  ClusterLayout C;
  std::memset(&C.P, 0, sizeof(C.P));
  TailPlan& P = C.P;
  int cf = std::max(H.coarse_from, from + 1);
  while (cf < H.levels - 1 && H.L[cf].cells > block_cells(H.dim)) ++cf;
  if (cf >= H.levels || cf - from > kMaxTail || H.levels - cf > kMaxCoarse) return C;
  P.count = cf - from;
  P.nu = W.nu;
  P.r_glob = r_glob;
  P.x_glob = x_glob;
  int off = kPlanWords;
  auto take = [&](int64_t n) {
    const int o = off;
    off += (int)up4(n);
    return o;
  };
  const MgLevel& M = H.L[cf];
  P.ep = (M.n[2] + res::kMaxCluster - 1) / res::kMaxCluster;
  P.C = lv(M);
  P.cdx = res::fast_div(M.n[0]);
  P.cdy = res::fast_div(M.n[1]);
  // a window: planes + 2 halos, padded by a row and a cell for the reads
  // across the domain's x and y edges
  auto window = [&](const MgLevel& L, int planes, int words) {
    const int64_t pad = (int64_t)up4(L.n[0] + 1) * words;
    const int64_t body = (int64_t)(planes + 2) * L.n[0] * L.n[1] * words;
    const int o = take(body + 2 * pad);
    return o + (int)pad;
  };
  int64_t total = 0;
  for (int q = 0; q < P.count; ++q) {
    const MgLevel& L = H.L[from + q];
    TailLevel& V = P.lv[q];
    V.L = lv(L);
    V.dx = res::fast_div(L.n[0]);
    V.dy = res::fast_div(L.n[1]);
    V.planes = P.ep << (P.count - q);
    V.K = kern_of(W, from + q);
    V.cw = cw_of(W, from + q);
    const int64_t own = (int64_t)V.planes * L.n[0] * L.n[1];
    total += 4 * own;
    if (total * (fcg && q == 0 ? 4 : 1) > (int64_t)res::kSmemMax) return C;  // (no overflow below)
    if (fcg && q == 0) {
      P.op = window(L, V.planes, 2);
      P.or64 = take(2 * own);
      P.oq = take(2 * own);
    } else {
      V.orr = take(own);
    }
    V.ox = window(L, V.planes, 1);
    V.ou = window(L, V.planes, 1);
  }
  P.oe = window(M, P.ep, 1);
  P.coarse = take((int64_t)(coarse_bytes(H, cf) / sizeof(float)));
  P.ox64 = -1;
  if (fcg) {
    const int64_t own = 2 * (int64_t)P.lv[0].planes * H.L[from].n[0] * H.L[from].n[1];
    if ((off + own) * 4 <= (int64_t)res::kSmemMax) P.ox64 = take(own);
  }
  if ((size_t)off * 4 > res::kSmemMax) return C;
  C.Q = coarse_plan(H, W, cf, kClusterT);
  C.words = off;
  return C;
}
