// Krylov solves whose vectors stay on chip.
//
// The streaming solvers (pcg_tma.cuh, stencil_krylov.cuh) move every vector
// through L2 once or more per iteration and cross the whole GPU in grid
// barriers built on one atomic counter.  A system that fits the chip needs
// neither: here every block owns one contiguous range of cells for the whole
// solve, keeps the vectors of its cells in shared memory and registers, and
// an iteration only exchanges the values of p at the ends of the ranges and
// the partial sums of the dot products.  What is left is the latency of the
// dependent steps: p -> A p -> alpha -> r -> beta.
//
// Two teams of blocks run the same routines:
//   ClusterTeam  one thread-block cluster of 1..16 blocks.  Neighbours read
//                each other's values in distributed shared memory, partial sums
//                are pushed into every block's shared memory, and the barrier is
//                the hardware cluster barrier.
//   GridTeam     one block per SM, cooperatively launched.  Values are
//                published in global memory (L2); a reduction is one release-
//                add on a counter and one acquiring poll (bounded) by one thread
//                per block, then every block adds all partial sums: 2.2 us with
//                148 blocks of 512 threads (an all-to-all exchange of tagged
//                values, polled without a counter, took 3.7 to 5.5 us for two
//                values: the polls contend with the writes).
//
// All sums run in a fixed order (threads by shuffle, warps, then blocks by
// rank), so a result does not depend on timing, and every block derives
// bitwise-identical scalars and takes the same branch.
#pragma once

#include <cuda_runtime.h>

#include <cfloat>
#include <cmath>
#include <cstdint>

#include "cell_index.cuh"
#include "cfdb.h"
#include "grid_sync.cuh"
#include "poperator.cuh"
#include "stencil_solve.cuh"

namespace cfdb {
namespace res {

// Couplings of one cell to its neighbours (0 across the domain's edge), its
// diagonal and the preconditioner's inverse diagonal.
template <typename V>
struct Cf {
  V xl, xh, yl, yh, zl, zh, dg, inv;
};

// ------------------------------------------------------------------ operators
//
// An operator has the extents of kernel space (a 2D grid is nx x 1 x ny),
// load() -> Cf of a cell and mul() -> the row's product; V is the type of its
// vectors and coefficients.

// The p' operator (poperator.cuh), tables or face arrays; Jacobi.
template <int DIM, typename T = double>
struct FaceOp {
  static constexpr int kDim = DIM;
  using V = T;
  OpView<V> A;
  const V* invd;  // 1/diag of face-array operators, or null
  int nx, ny, nz;
  uint32_t sz;
  FastDiv dx, dy;
  __device__ __forceinline__ Cf<V> load(uint32_t c, int i, int j, int k) const {
    Cf<V> f;
    const uint32_t row = (uint32_t)j + (uint32_t)ny * k;
    if (A.fx) {
      f.xl = __ldg(A.fx + c + row);
      f.xh = __ldg(A.fx + c + row + 1);
    } else {
      f.xl = __ldg(A.tx + i);
      f.xh = __ldg(A.tx + i + 1);
    }
    f.yl = f.yh = V(0);
    if (DIM == 3) {
      if (A.fy) {
        f.yl = __ldg(A.fy + c + (uint32_t)nx * k);
        f.yh = __ldg(A.fy + c + (uint32_t)nx * k + nx);
      } else {
        f.yl = __ldg(A.ty + j);
        f.yh = __ldg(A.ty + j + 1);
      }
    }
    if (A.fz) {
      f.zl = __ldg(A.fz + c);
      f.zh = __ldg(A.fz + c + sz);
    } else {
      f.zl = __ldg(A.tz + k);
      f.zh = __ldg(A.tz + k + 1);
    }
    if (A.pinned && c == (uint32_t)A.ref) {
      f.xl = f.xh = f.yl = f.yh = f.zl = f.zh = V(0);
      f.dg = f.inv = V(1);
      return f;
    }
    // the reference's face order (poperator.cuh load_coef)
    f.dg = ((((f.xl + f.xh) + f.yl) + f.yh) + f.zl) + f.zh;
    f.inv = invd ? __ldg(invd + c) : rcp_rn(f.dg);
    if (i == 0) f.xl = V(0);
    if (i == nx - 1) f.xh = V(0);
    if (j == 0) f.yl = V(0);
    if (j == ny - 1) f.yh = V(0);
    if (k == 0) f.zl = V(0);
    if (k == nz - 1) f.zh = V(0);
    return f;
  }
  // the preconditioner's inverse diagonal alone
  __device__ __forceinline__ V inverse(uint32_t c, int i, int j, int k) const {
    if (invd) return __ldg(invd + c);
    if (A.fx || A.fy || A.fz) return load(c, i, j, k).inv;
    if (A.pinned && c == (uint32_t)A.ref) return V(1);
    V d = __ldg(A.tx + i) + __ldg(A.tx + i + 1);
    if (DIM == 3) d = (d + __ldg(A.ty + j)) + __ldg(A.ty + j + 1);
    return rcp_rn((d + __ldg(A.tz + k)) + __ldg(A.tz + k + 1));
  }
  __device__ __forceinline__ V mul(const Cf<V>& f, V v, V w, V e, V s, V n, V b, V t) const {
    V off = f.xl * w;
    off = fma(f.xh, e, off);
    if (DIM == 3) {
      off = fma(f.yl, s, off);
      off = fma(f.yh, n, off);
    }
    off = fma(f.zl, b, off);
    off = fma(f.zh, t, off);
    return fma(f.dg, v, -off);
  }
};

template <int DIM, typename V>
__host__ __device__ inline FaceOp<DIM, V> face_op(const OpView<V>& A, const V* invd) {
  FaceOp<DIM, V> f;
  f.A = A;
  f.invd = invd;
  f.nx = A.nx;
  f.ny = A.ny;
  f.nz = A.nz;
  f.sz = (uint32_t)A.nx * A.ny;
  f.dx = fast_div(A.nx);
  f.dy = fast_div(A.ny);
  return f;
}

// A stored stencil matrix (stencil_solve.cuh); inv null: no preconditioner.
// A 2D matrix's second axis is kernel space's z.
template <int DIM>
struct BandOp {
  static constexpr int kDim = DIM;
  using V = double;
  const double* diag;
  const double *oxl, *oxh, *oyl, *oyh, *ozl, *ozh;
  const double* pinv;
  int nx, ny, nz;
  uint32_t sz;
  FastDiv dx, dy;
  __device__ __forceinline__ Cf<double> load(uint32_t c, int i, int j, int k) const {
    Cf<double> f;
    f.xl = i > 0 ? __ldg(oxl + c) : 0.0;
    f.xh = i < nx - 1 ? __ldg(oxh + c) : 0.0;
    f.yl = DIM == 3 && j > 0 ? __ldg(oyl + c) : 0.0;
    f.yh = DIM == 3 && j < ny - 1 ? __ldg(oyh + c) : 0.0;
    f.zl = k > 0 ? __ldg(ozl + c) : 0.0;
    f.zh = k < nz - 1 ? __ldg(ozh + c) : 0.0;
    f.dg = __ldg(diag + c);
    f.inv = pinv ? __ldg(pinv + c) : 1.0;
    return f;
  }
  __device__ __forceinline__ double inverse(uint32_t c, int, int, int) const {
    return pinv ? __ldg(pinv + c) : 1.0;
  }
  // ascending column order of the reference's CSR rows
  __device__ __forceinline__ double mul(const Cf<double>& f, double v, double w, double e, double s,
                                        double n, double b, double t) const {
    double sum = f.zl * b;
    if (DIM == 3) sum += f.yl * s;
    sum += f.xl * w;
    sum += f.dg * v;
    sum += f.xh * e;
    if (DIM == 3) sum += f.yh * n;
    sum += f.zh * t;
    return sum;
  }
};

template <int DIM>
__host__ __device__ inline BandOp<DIM> band_op(const StencilMatrix& M) {
  BandOp<DIM> A;
  A.oyl = A.oyh = nullptr;
  A.diag = M.diag;
  A.oxl = M.off[0];
  A.oxh = M.off[1];
  if (DIM == 3) {
    A.oyl = M.off[2];
    A.oyh = M.off[3];
    A.ozl = M.off[4];
    A.ozh = M.off[5];
  } else {
    A.ozl = M.off[2];
    A.ozh = M.off[3];
  }
  A.pinv = M.inv;
  A.nx = M.nx;
  A.ny = DIM == 3 ? M.ny : 1;
  A.nz = DIM == 3 ? M.nz : M.ny;
  A.sz = (uint32_t)A.nx * A.ny;
  A.dx = fast_div(A.nx);
  A.dy = fast_div(A.ny);
  return A;
}

// ---------------------------------------------------------------------- teams

constexpr int kMaxCluster = 16;
constexpr int kMaxVals = 3;

// Sum of N values of an array by halves (fixed order; N a power of two).
template <int N>
__device__ __forceinline__ double tree(double (&a)[N]) {
#pragma unroll
  for (int w = N / 2; w > 0; w >>= 1)
#pragma unroll
    for (int s = 0; s < w; ++s) a[s] += a[s + w];
  return a[0];
}

// Block-wide sum in a fixed order, valid in every thread of warp 0 (`W`
// warps, a power of two).  The warps' sums are added from shared memory by a
// tree in registers: half the latency of a second round of shuffles.
template <int NV, int W>
__device__ __forceinline__ void block_total(double (&v)[NV], double (*red)[32]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NV; ++q)
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], off);
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < NV; ++q) red[q][warp] = v[q];
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      double a[W];
#pragma unroll
      for (int s = 0; s < W; ++s) a[s] = red[q][s];
      v[q] = tree<W>(a);
    }
  }
}

struct TeamSmem {
  alignas(16) double red[kMaxVals][32];
  alignas(16) double slot[2][kMaxVals][kMaxCluster];  // cluster: every block's sums, by parity
  alignas(16) double poll[kMaxVals][8];               // grid: the polling warps' sums
};

template <int T>
struct ClusterTeam {
  static constexpr bool kGlobal = false;
  int rank_, size_;
  int parity = 0;
  FastDiv dlen;
  uint32_t len;
  TeamSmem* ts;
  __device__ int rank() const { return rank_; }
  __device__ __forceinline__ bool sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;"
                 ::: "memory");
    return true;
  }
  // Before a block's first store into another's shared memory (a reduction
  // makes one): every block of the cluster has started.
  __device__ __forceinline__ void enter() { sync(); }
  // The team-wide sums of v, in every thread; a full barrier of the team.
  template <int NV>
  __device__ __forceinline__ bool reduce(double (&v)[NV]) {
    block_total<NV, T / 32>(v, ts->red);
    if ((int)threadIdx.x < size_) {
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        const uint32_t a = (uint32_t)__cvta_generic_to_shared(&ts->slot[parity][q][rank_]);
        uint32_t ra;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(threadIdx.x));
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(ra), "d"(v[q]) : "memory");
      }
    }
    sync();
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      double a[kMaxCluster];
#pragma unroll
      for (int s = 0; s < kMaxCluster; ++s) a[s] = s < size_ ? ts->slot[parity][q][s] : 0.0;
      v[q] = tree<kMaxCluster>(a);
    }
    parity ^= 1;
    return true;
  }
  // vec[c] of a cell outside this block's range (vec: this block's shared array)
  __device__ __forceinline__ float remote(const float* vec, const float*, uint32_t c) const {
    const uint32_t r = dlen.div(c);
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(vec + (c - r * len));
    uint32_t ra;
    float out;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(r));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(out) : "r"(ra) : "memory");
    return out;
  }
  __device__ __forceinline__ double remote(const double* vec, const double*, uint32_t c) const {
    const uint32_t r = dlen.div(c);
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(vec + (c - r * len));
    uint32_t ra;
    double out;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(r));
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(out) : "r"(ra) : "memory");
    return out;
  }
};

template <int T>
struct GridTeam {
  static constexpr bool kGlobal = true;
  static constexpr int kPollers = 256;  // threads that read the partial sums: >= blocks
  static_assert(T >= kPollers, "one thread per block reads its partial sums");
  double* partials;  // 2 parities x blocks x kMaxVals
  unsigned* count;   // arrivals since the launch (wraps)
  unsigned* error;
  unsigned long long timeout_ns;
  int rank_, size_;
  unsigned round = 0;
  TeamSmem* ts;
  __device__ int rank() const { return rank_; }
  // Thread 0 arrives (after a block barrier: its release covers the whole
  // block's stores) and waits, bounded, for every block of this round.
  __device__ __forceinline__ bool arrive_and_wait() {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
    const unsigned target = round * (unsigned)size_;
    unsigned long long t0 = 0;
    for (unsigned spin = 0;; ++spin) {
      unsigned c;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(count) : "memory");
      if ((int)(c - target) >= 0) return *(volatile unsigned*)error == 0u;
      if ((spin & 63u) != 63u) continue;
      const unsigned long long now = global_ns();
      if (t0 == 0) t0 = now;
      if (*(volatile unsigned*)error != 0u) return false;
      if (now - t0 > timeout_ns) {
        atomicExch(error, 1u);
        return false;
      }
    }
  }
  // Global memory needs no block to have started.
  __device__ __forceinline__ void enter() {}
  // published values are visible to every block afterwards
  __device__ __forceinline__ bool sync() {
    ++round;
    __syncthreads();
    bool ok = true;
    if (threadIdx.x == 0) ok = arrive_and_wait();
    return __syncthreads_and(ok);
  }
  // The team-wide sums of v, in every thread; a full barrier of the team.
  template <int NV>
  __device__ __forceinline__ bool reduce(double (&v)[NV]) {
    block_total<NV, T / 32>(v, ts->red);
    ++round;
    double* base = partials + (size_t)(round & 1) * size_ * kMaxVals;
    const int t = threadIdx.x;
    bool ok = true;
    if (t == 0) {
#pragma unroll
      for (int q = 0; q < NV; ++q) __stcg(base + rank_ * NV + q, v[q]);
      ok = arrive_and_wait();
    }
    if (!__syncthreads_and(ok)) return false;
    if (t < kPollers) {
      double a[NV];
#pragma unroll
      for (int q = 0; q < NV; ++q) a[q] = t < size_ ? __ldcg(base + t * NV + q) : 0.0;
#pragma unroll
      for (int q = 0; q < NV; ++q)
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) a[q] += __shfl_xor_sync(0xffffffffu, a[q], off);
      if ((t & 31) == 0)
#pragma unroll
        for (int q = 0; q < NV; ++q) ts->poll[q][t >> 5] = a[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      double b[kPollers / 32];
#pragma unroll
      for (int s = 0; s < kPollers / 32; ++s) b[s] = ts->poll[q][s];
      v[q] = tree<kPollers / 32>(b);
    }
    return true;
  }
  template <typename V>
  __device__ __forceinline__ V remote(const V*, const V* pub, uint32_t c) const {
    return __ldcg(pub + c);
  }
};

// ------------------------------------------------------------------- routines

template <typename V>
struct IoT {
  const V* b;
  V* x;
  V* pub;   // GridTeam: published values (cells), else null
  V* pub2;  // GridTeam, BiCGSTAB: published s (cells)
  V* inv;   // scratch (cells) for M^-1 of a table operator, or null
  double abs_tol, rel_tol;
  int64_t max_it;
  double* hist;
  int64_t hist_cap;
  double* out;   // status, iterations, initial residual, final residual, restarts
  double delta;  // MIXED: drop of the residual between replacements
  double* reps;  // MIXED: where the number of replacements goes
};
using Io = IoT<double>;

// Range of cells of block `rank`: [rank len, min(n, (rank + 1) len)).
struct Range {
  uint32_t c0, count;
};
__device__ __forceinline__ Range range_of(uint32_t n, uint32_t len, int rank) {
  const uint32_t c0 = min(n, len * (uint32_t)rank);
  return Range{c0, min(len, n - c0)};
}

// The coefficients of a thread's NC cells: kept in registers for the whole
// solve when there are few of them, else loaded again where they are used.
template <class Op, int NC, bool PRE>
struct Cells {
  using V = typename Op::V;
  Cf<V> f[PRE ? NC : 1];
  __device__ __forceinline__ void ijk(const Op& A, uint32_t c, int& i, int& j, int& k) const {
    const uint32_t row = A.dx.div(c);
    i = (int)(c - row * (uint32_t)A.nx);
    if (Op::kDim == 3) {
      const uint32_t kk = A.dy.div(row);
      k = (int)kk;
      j = (int)(row - kk * (uint32_t)A.ny);
    } else {
      k = (int)row;
      j = 0;
    }
  }
  __device__ __forceinline__ Cf<V> load(const Op& A, uint32_t c) const {
    int i, j, k;
    ijk(A, c, i, j, k);
    return A.load(c, i, j, k);
  }
  template <int T>
  __device__ __forceinline__ void init(const Op& A, const Range& R) {
    if constexpr (PRE) {
#pragma unroll
      for (int q = 0; q < NC; ++q) {
        const uint32_t lc = threadIdx.x + q * T;
        if (lc < R.count) f[q] = load(A, R.c0 + lc);
      }
    }
  }
  __device__ __forceinline__ Cf<V> at(const Op& A, int q, uint32_t c) const {
    if constexpr (PRE) return f[q];
    else return load(A, c);
  }
  __device__ __forceinline__ V inverse(const Op& A, int q, uint32_t c) const {
    if constexpr (PRE) return f[q].inv;
    int i, j, k;
    ijk(A, c, i, j, k);
    return A.inverse(c, i, j, k);
  }
};

// (A v)(c) with v in this block's shared array.  HALO: every neighbour is in
// the array.  Else x- and y-neighbours past the range's ends are read from
// the published vector (couplings of 0 read nothing), and the z-neighbours'
// values come with the call.
template <bool HALO, class Op, class Team, typename V = typename Op::V>
__device__ __forceinline__ V apply(const Op& A, const Team& T, const Cf<V>& f, const Range& R,
                                   uint32_t lc, const V* vec, const V* pub, V zlo, V zhi) {
  const int sy = A.nx, sz = (int)A.sz;
  const V* v = vec + lc;
  if constexpr (HALO) {
    return A.mul(f, v[0], v[-1], v[1], Op::kDim == 3 ? v[-sy] : V(0), Op::kDim == 3 ? v[sy] : V(0),
                 v[-sz], v[sz]);
  } else {
    const uint32_t c = R.c0 + lc;
    auto get = [&](V coupling, int off) -> V {
      const uint32_t li = lc + (uint32_t)off;  // wraps below 0: past count
      if (li < R.count) return vec[li];
      return coupling == V(0) ? V(0) : T.remote(vec, pub, c + (uint32_t)off);
    };
    return A.mul(f, v[0], get(f.xl, -1), get(f.xh, 1), Op::kDim == 3 ? get(f.yl, -sy) : V(0),
                 Op::kDim == 3 ? get(f.yh, sy) : V(0), zlo, zhi);
  }
}

// (A x)(c) with x in global memory.
template <class Op, typename V = typename Op::V>
__device__ __forceinline__ V apply_global(const Op& A, const Cf<V>& f, uint32_t c, const V* x) {
  auto get = [&](V coupling, uint32_t at) { return coupling == V(0) ? V(0) : __ldcg(x + at); };
  const uint32_t sy = (uint32_t)A.nx, sz = A.sz;
  return A.mul(f, __ldcg(x + c), get(f.xl, c - 1), get(f.xh, c + 1),
               Op::kDim == 3 ? get(f.yl, c - sy) : V(0), Op::kDim == 3 ? get(f.yh, c + sy) : V(0),
               get(f.zl, c - sz), get(f.zh, c + sz));
}

// Jacobi-CG (or plain CG), the reference's method and tests (CG.cpp:14-148).
//
// HALO: the block also keeps p of the H = one plane (2D: row) of cells before
// and after its range, and forms it there as its owners do, from the
// published z = M^-1 r and its own old p; an iteration then has two exchanges
// (the two reductions).  Otherwise (3D grids whose planes are larger than
// shared memory allows) p itself is published, which takes a third.
//
// MIXED (V = double): the mixed-precision solve of pcg_tma.cuh -- z and p are
// rounded to FP32 as they are formed, x and r stay FP64 and r is replaced by
// b - A x when it has fallen by P.delta, when it meets the tolerance and at
// the iteration cap.
//
// Shared memory (words of V): p (len, HALO: + 2 H), r (len), ClusterTeam: z
// (len), XS: x (len).
template <int T, int NC, bool PRE, bool XS, bool HALO, bool MIXED = false, class Op, class Team,
          typename V = typename Op::V>
__device__ __forceinline__ void cg_run(const Op& A, uint32_t n, uint32_t len, const IoT<V>& P,
                                       Team& team, V* sm) {
  static_assert(HALO || Team::kGlobal, "a cluster's planes fit its shared memory");
  const Range R = range_of(n, len, team.rank());
  const uint32_t H = A.sz;  // reach of the stencil
  V* p = HALO ? sm + H : sm;
  V* r = sm + len + (HALO ? 2 * H : 0);
  V* zs = r + len;
  V* xs = zs + (Team::kGlobal ? 0 : len);
  const bool leader = team.rank() == 0 && threadIdx.x == 0;
  Cells<Op, NC, PRE> cells;
  cells.template init<T>(A, R);
  if (HALO)
    for (uint32_t q = threadIdx.x; q < len + 2 * H; q += T) sm[q] = V(0);
  team.enter();
  V z[NC];  // z = M^-1 r between the sweeps, q = A p within an iteration
  // z of a cell for the blocks whose stencils reach it
  auto rounded = [](V v) { return MIXED ? (V)(float)v : v; };
  // p = z + beta p_old
  auto direction = [](V beta, V old, V zv) {
    return MIXED ? (V)fmaf((float)beta, (float)old, (float)zv) : fma(beta, old, zv);
  };
  auto publish = [&](uint32_t lc, V v) {
    if (!Team::kGlobal) zs[lc] = v;
    else if (!HALO || lc < H || lc + H >= R.count) P.pub[R.c0 + lc] = v;
  };
  // r = b - A x (x in global memory), z = M^-1 r; r.r, r.z
  auto residual = [&](double (&acc)[2]) -> bool {
    acc[0] = acc[1] = 0.0;
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      const uint32_t lc = threadIdx.x + q * T;
      if (lc < R.count) {
        const uint32_t c = R.c0 + lc;
        const Cf<V> f = cells.at(A, q, c);
        const V rn = __ldg(P.b + c) - apply_global(A, f, c, P.x);
        r[lc] = rn;
        z[q] = rounded(f.inv * rn);
        if (HALO) publish(lc, z[q]);
        if (!PRE && P.inv) P.inv[c] = f.inv;
        acc[0] += (double)rn * (double)rn;
        acc[1] += (double)rn * (double)z[q];
      }
    }
    return team.reduce(acc);
  };
  auto flush_x = [&]() {
    if (XS) {
#pragma unroll
      for (int q = 0; q < NC; ++q) {
        const uint32_t lc = threadIdx.x + q * T;
        if (lc < R.count) P.x[R.c0 + lc] = xs[lc];
      }
    }
  };
  double acc[2];
  if (XS) {
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      const uint32_t lc = threadIdx.x + q * T;
      if (lc < R.count) xs[lc] = __ldcg(P.x + R.c0 + lc);
    }
  }
  if (!residual(acc)) return;
  const double b0 = sqrt(acc[0]);
  double rz = acc[1];
  auto conv = [&](double res) {
    return (res <= P.abs_tol) || ((b0 > 0.0) && (res / b0 <= P.rel_tol));
  };
  auto finish = [&](int status, int64_t it, double fin) {
    if (leader) {
      P.out[0] = status;
      P.out[1] = (double)it;
      P.out[3] = fin;
    }
    if (it > 0) flush_x();
  };
  if (leader) {
    P.out[2] = b0;
    P.out[4] = 0.0;
    if (MIXED) *P.reps = 0.0;
    if (P.hist_cap > 0) P.hist[0] = b0;
  }
  if (b0 == 0.0 || conv(b0)) return finish(CFDB_SOLVER_CONVERGED, 0, b0);
  if (!isfinite(rz)) return finish(CFDB_SOLVER_BREAKDOWN, 0, b0);
  // cells of the halo inside the domain: [lo0, c0) and [c0 + count, hi1)
  const uint32_t lo = min(H, R.c0), hi = min(H, n - (R.c0 + R.count));
  double res_cur = b0, beta = 0.0, replaced = b0;
  int64_t reps = 0;
  for (int64_t it = 1; it <= P.max_it; ++it) {
    // p = z + beta p
    if (HALO && R.count > 0) {
      for (uint32_t h = threadIdx.x; h < lo + hi; h += T) {
        const int at = h < lo ? -(int)(lo - h) : (int)(R.count + (h - lo));
        p[at] = direction((V)beta, p[at], team.remote(zs, P.pub, R.c0 + (uint32_t)at));
      }
    }
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      const uint32_t lc = threadIdx.x + q * T;
      if (lc < R.count) {
        const V v = it == 1 ? z[q] : direction((V)beta, p[lc], z[q]);
        p[lc] = v;
        if (!HALO) publish(lc, v);
      }
    }
    if (HALO) __syncthreads();
    else if (!team.sync()) return;
    double pap[1] = {0.0};
    if constexpr (HALO) {
#pragma unroll
      for (int q = 0; q < NC; ++q) {
        const uint32_t lc = threadIdx.x + q * T;
        if (lc < R.count) {
          const Cf<V> f = cells.at(A, q, R.c0 + lc);
          z[q] = apply<true>(A, team, f, R, lc, p, P.pub, V(0), V(0));
          pap[0] += (double)p[lc] * (double)z[q];
        }
      }
    } else {
      // the z-neighbours of a batch of cells, all from L2, are loaded before
      // the first is used
      constexpr int G = NC % 4 == 0 ? 4 : (NC % 2 == 0 ? 2 : 1);
#pragma unroll
      for (int g = 0; g < NC; g += G) {
        V lo_z[G], hi_z[G];
#pragma unroll
        for (int u = 0; u < G; ++u) {
          const uint32_t c = R.c0 + threadIdx.x + (g + u) * T;
          const bool in = threadIdx.x + (g + u) * T < R.count;
          lo_z[u] = in && c >= H ? __ldcg(P.pub + (c - H)) : V(0);
          hi_z[u] = in && c + H < n ? __ldcg(P.pub + (c + H)) : V(0);
        }
#pragma unroll
        for (int u = 0; u < G; ++u) {
          const int q = g + u;
          const uint32_t lc = threadIdx.x + q * T;
          if (lc < R.count) {
            const Cf<V> f = cells.at(A, q, R.c0 + lc);
            z[q] = apply<false>(A, team, f, R, lc, p, P.pub, lo_z[u], hi_z[u]);
            pap[0] += (double)p[lc] * (double)z[q];
          }
        }
      }
    }
    if (!team.reduce(pap)) return;
    const double pAp = pap[0];
    const double alpha = rz / pAp;
    if (!isfinite(pAp) || fabs(pAp) < 1.0e-30 || !isfinite(alpha))
      return finish(CFDB_SOLVER_BREAKDOWN, it - 1, res_cur);
    double ab[2] = {0.0, 0.0};
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      const uint32_t lc = threadIdx.x + q * T;
      if (lc < R.count) {
        if (XS) xs[lc] = fma((V)alpha, p[lc], xs[lc]);
        else P.x[R.c0 + lc] = fma((V)alpha, p[lc], P.x[R.c0 + lc]);
        const V rn = fma(-(V)alpha, z[q], r[lc]);
        r[lc] = rn;
        z[q] = rounded((!PRE && P.inv ? P.inv[R.c0 + lc] : cells.inverse(A, q, R.c0 + lc)) * rn);
        if (HALO) publish(lc, z[q]);
        ab[0] += (double)rn * (double)rn;
        ab[1] += (double)rn * (double)z[q];
      }
    }
    if (!team.reduce(ab)) return;
    double res = sqrt(ab[0]);
    if (MIXED && isfinite(res) && (conv(res) || res <= P.delta * replaced || it == P.max_it)) {
      flush_x();
      if (!team.sync()) return;  // x of every block is in memory
      if (!residual(ab)) return;
      res = replaced = sqrt(ab[0]);
      ++reps;
      if (leader) *P.reps = (double)reps;
    }
    if (leader && it < P.hist_cap) P.hist[it] = res;
    if (!isfinite(res)) return finish(CFDB_SOLVER_NONFINITE_RESIDUAL, it, res);
    res_cur = res;
    if (conv(res)) return finish(CFDB_SOLVER_CONVERGED, it, res);
    beta = ab[1] / rz;
    if (!isfinite(ab[1]) || !isfinite(beta)) return finish(CFDB_SOLVER_BREAKDOWN, it, res);
    rz = ab[1];
  }
  finish(CFDB_SOLVER_MAX_ITERATIONS, P.max_it, res_cur);
}

// (A v^)(c), v^ = v (or, PREC, M^-1 v), v in this block's shared array and,
// past the range's ends, published by the team; the z-neighbours come with
// the call (see gather_z).
template <bool PREC, class Op, class Team>
__device__ __forceinline__ double neighbour(const Op& A, const Team& T, double coupling,
                                            const Range& R, uint32_t lc, int off,
                                            const double* vec, const double* pub) {
  if (coupling == 0.0) return 0.0;
  const uint32_t li = lc + (uint32_t)off, c = R.c0 + lc + (uint32_t)off;
  const double v = li < R.count ? vec[li] : T.remote(vec, pub, c);
  return PREC ? v * __ldg(A.pinv + c) : v;
}

// out = A v^ for the thread's cells.  The z-neighbours of two cells
// are read before the first is used: in 3D they are all outside the block's
// range, one trip through the team each.  NC > 0: at most NC cells a thread,
// their coefficients in registers; NC = 0: any number.
template <int T, int NC, bool PREC, class Op, class Team>
__device__ __forceinline__ void spmv(const Op& A, const Cells<Op, NC ? NC : 1, (NC > 0)>& cells,
                                     const Range& R, const Team& team, const double* vec,
                                     const double* pub, double* out) {
  constexpr int G = NC ? NC : 2;
  const int sy = A.nx, sz = (int)A.sz;
  for (uint32_t g = threadIdx.x; g < R.count; g += G * T) {
    Cf<double> f[G];
    double lo[G], hi[G];
#pragma unroll
    for (int u = 0; u < G; ++u) {
      const uint32_t lc = g + u * T;
      if (lc < R.count) {
        f[u] = cells.at(A, NC ? u : 0, R.c0 + lc);
        lo[u] = neighbour<PREC>(A, team, f[u].zl, R, lc, -sz, vec, pub);
        hi[u] = neighbour<PREC>(A, team, f[u].zh, R, lc, sz, vec, pub);
      }
    }
#pragma unroll
    for (int u = 0; u < G; ++u) {
      const uint32_t lc = g + u * T;
      if (lc < R.count)
        out[lc] = A.mul(
            f[u], PREC ? vec[lc] * f[u].inv : vec[lc],
            neighbour<PREC>(A, team, f[u].xl, R, lc, -1, vec, pub),
            neighbour<PREC>(A, team, f[u].xh, R, lc, 1, vec, pub),
            Op::kDim == 3 ? neighbour<PREC>(A, team, f[u].yl, R, lc, -sy, vec, pub) : 0.0,
            Op::kDim == 3 ? neighbour<PREC>(A, team, f[u].yh, R, lc, sy, vec, pub) : 0.0, lo[u], hi[u]);
    }
  }
}

// BiCGSTAB with the reference's breakdown and restart tests
// (BiCGSTAB.cpp:48-275), the arithmetic of krylov_run (stencil_krylov.cuh).
// The ranges' ends exchange p once (a barrier of its own) and s (with the
// reduction of |s|^2): five barriers an iteration, four of them reductions.
// Shared memory (doubles): p, r/s, rHat, v, t and (XS) x, len each.  The
// loops over a thread's cells stay rolled unless there are at most two: fully
// unrolled, the addresses of every cell are kept across the iteration and
// spill.
template <int T, int NC, bool XS, bool PREC, class Op, class Team>
__device__ __forceinline__ void bicgstab_run(const Op& A, uint32_t n, uint32_t len, const Io& P,
                                             Team& team, double* sm) {
  const Range R = range_of(n, len, team.rank());
  double* p = sm;
  double* r = sm + len;  // r, and s between the half steps
  double* rh = sm + 2 * (size_t)len;
  double* v = sm + 3 * (size_t)len;
  double* t = sm + 4 * (size_t)len;
  double* xs = sm + 5 * (size_t)len;
  const uint32_t H = A.sz;
  const bool leader = team.rank() == 0 && threadIdx.x == 0;
  Cells<Op, NC ? NC : 1, (NC > 0)> cells;
  cells.template init<T>(A, R);
  auto each = [&](auto f) {
    if constexpr (NC > 0) {
#pragma unroll
      for (int q = 0; q < NC; ++q) {
        const uint32_t lc = threadIdx.x + q * T;
        if (lc < R.count) f(q, lc, R.c0 + lc);
      }
    } else {
#pragma unroll 2
      for (uint32_t lc = threadIdx.x; lc < R.count; lc += T) f(0, lc, R.c0 + lc);
    }
  };
  auto publish = [&](double* pub, uint32_t lc, double val) {
    if (Team::kGlobal && (lc < H || lc + H >= R.count)) pub[R.c0 + lc] = val;
  };
  auto x_at = [&](uint32_t lc) { return XS ? xs[lc] : P.x[R.c0 + lc]; };
  auto set_x = [&](uint32_t lc, double val) {
    if (XS) xs[lc] = val;
    else P.x[R.c0 + lc] = val;
  };
  auto flush_x = [&]() {
    if (XS) each([&](int, uint32_t lc, uint32_t c) { P.x[c] = xs[lc]; });
  };
  auto finish = [&](int status, int64_t it, double fin) {
    if (leader) {
      P.out[0] = status;
      P.out[1] = (double)it;
      P.out[3] = fin;
    }
    flush_x();
  };
  const double eps = DBL_EPSILON;
  auto cancelled = [&](double ip, double nx_, double ny_, double terms) {
    if (fabs(ip) > eps * nx_ * ny_) return false;
    return fabs(ip) <= eps * terms;
  };
  // r = rHat = b - A x (x in global memory), v = p = 0; (r, r)
  auto start = [&](double (&o)[1]) -> bool {
    o[0] = 0.0;
    each([&](int q, uint32_t lc, uint32_t c) {
      const Cf<double> f = cells.at(A, q, c);
      const double rn = __ldg(P.b + c) - apply_global(A, f, c, P.x);
      r[lc] = rn;
      rh[lc] = rn;
      v[lc] = 0.0;
      p[lc] = 0.0;
      o[0] += rn * rn;
    });
    return team.reduce(o);
  };
  if (XS) each([&](int, uint32_t lc, uint32_t c) { xs[lc] = __ldcg(P.x + c); });
  team.enter();
  double tot[3], one[1];
  if (!start(one)) return;
  const double b0 = sqrt(one[0]);
  if (leader) {
    P.out[2] = b0;
    P.out[4] = 0.0;
    if (P.hist_cap > 0) P.hist[0] = b0;
  }
  auto conv = [&](double res) {
    return (res <= P.abs_tol) || ((b0 > 0.0) && (res / b0 <= P.rel_tol));
  };
  if (b0 == 0.0 || conv(b0)) return finish(CFDB_SOLVER_CONVERGED, 0, b0);
  double rhoOld = 1.0, alpha = 1.0, omega = 1.0;
  int64_t completed = 0, restarts = 0, hc = 1;
  double rHatNorm = b0, rNorm = b0, restartResidual = b0, lastHist = b0;
  double rho = one[0], rhoTerms = one[0];
  auto push = [&](double val) {
    if (leader && hc < P.hist_cap) P.hist[hc] = val;
    ++hc;
  };
  // restart (BiCGSTAB.cpp:127-151): 0 restarted, 1 converged, 2 stop
  auto restart = [&](int& outcome) -> bool {
    outcome = 2;
    if (!(rNorm < restartResidual)) return true;
    flush_x();
    if (!team.sync()) return false;
    double o[1];
    if (!start(o)) return false;
    rNorm = sqrt(o[0]);
    if (!isfinite(rNorm)) return true;
    if (conv(rNorm)) {
      outcome = 1;
      return true;
    }
    rHatNorm = rNorm;
    restartResidual = rNorm;
    rhoOld = 1.0;
    alpha = 1.0;
    omega = 1.0;
    rho = o[0];
    rhoTerms = o[0];
    ++restarts;
    if (leader) P.out[4] = (double)restarts;
    outcome = 0;
    return true;
  };
  while (completed < P.max_it) {
    const int64_t iter = completed + 1;
    if (!isfinite(rho)) return finish(CFDB_SOLVER_BREAKDOWN, completed, rNorm);
    int oc = 0;
    if (cancelled(rho, rHatNorm, rNorm, rhoTerms)) {
      if (!restart(oc)) return;
      if (oc == 0) continue;
      return finish(oc == 1 ? CFDB_SOLVER_CONVERGED : CFDB_SOLVER_BREAKDOWN, completed, rNorm);
    }
    const double beta = (rho / rhoOld) * (alpha / omega);
    if (!isfinite(beta)) return finish(CFDB_SOLVER_BREAKDOWN, completed, rNorm);
    // p = r + (p - v omega) beta
    each([&](int, uint32_t lc, uint32_t) {
      const double val = r[lc] + (p[lc] - v[lc] * omega) * beta;
      p[lc] = val;
      publish(P.pub, lc, val);
    });
    if (!team.sync()) return;
    // v = A p^; (rHat, v), |v|^2, sum |rHat_i v_i|
    tot[0] = tot[1] = tot[2] = 0.0;
    spmv<T, NC, PREC>(A, cells, R, team, p, P.pub, v);
    each([&](int, uint32_t lc, uint32_t) {
      const double rhv = rh[lc] * v[lc];
      tot[0] = fma(rh[lc], v[lc], tot[0]);  // one rounding, as in krylov_run
      tot[1] += v[lc] * v[lc];
      tot[2] += fabs(rhv);
    });
    if (!team.reduce(tot)) return;
    const double rHatDotV = tot[0];
    if (!isfinite(rHatDotV)) return finish(CFDB_SOLVER_BREAKDOWN, completed, rNorm);
    if (cancelled(rHatDotV, rHatNorm, sqrt(tot[1]), tot[2])) {
      if (!restart(oc)) return;
      if (oc == 0) continue;
      return finish(oc == 1 ? CFDB_SOLVER_CONVERGED : CFDB_SOLVER_BREAKDOWN, completed, rNorm);
    }
    alpha = rho / rHatDotV;
    if (!isfinite(alpha)) return finish(CFDB_SOLVER_BREAKDOWN, completed, rNorm);
    // s = r - v alpha; |s|^2
    one[0] = 0.0;
    each([&](int, uint32_t lc, uint32_t) {
      const double sv = r[lc] - v[lc] * alpha;
      r[lc] = sv;
      publish(P.pub2, lc, sv);
      one[0] += sv * sv;
    });
    if (!team.reduce(one)) return;
    const double sNorm = sqrt(one[0]);
    if (!isfinite(sNorm)) {
      push(sNorm);
      return finish(CFDB_SOLVER_NONFINITE_RESIDUAL, iter, sNorm);
    }
    if (conv(sNorm)) {
      each([&](int q, uint32_t lc, uint32_t c) {
        const double ph = PREC ? p[lc] * cells.inverse(A, q, c) : p[lc];
        set_x(lc, x_at(lc) + ph * alpha);
      });
      push(sNorm);
      return finish(CFDB_SOLVER_CONVERGED, iter, sNorm);
    }
    // t = A s^; t.t, t.s, sum |t_i s_i|
    tot[0] = tot[1] = tot[2] = 0.0;
    spmv<T, NC, PREC>(A, cells, R, team, r, P.pub2, t);
    each([&](int, uint32_t lc, uint32_t) {
      const double tsv = t[lc] * r[lc];
      tot[0] += t[lc] * t[lc];
      tot[1] = fma(t[lc], r[lc], tot[1]);
      tot[2] += fabs(tsv);
    });
    if (!team.reduce(tot)) return;
    const double tDotT = tot[0], tDotS = tot[1];
    if (!isfinite(tDotT) || tDotT < DBL_MIN) return finish(CFDB_SOLVER_BREAKDOWN, completed, rNorm);
    if (!isfinite(tDotS)) return finish(CFDB_SOLVER_BREAKDOWN, completed, rNorm);
    if (cancelled(tDotS, sqrt(tDotT), sNorm, tot[2])) {
      if (!restart(oc)) return;
      if (oc == 0) continue;
      return finish(oc == 1 ? CFDB_SOLVER_CONVERGED : CFDB_SOLVER_BREAKDOWN, completed, rNorm);
    }
    omega = tDotS / tDotT;
    if (!isfinite(omega)) return finish(CFDB_SOLVER_BREAKDOWN, completed, rNorm);
    // x += p^ alpha; x += s^ omega; r = s - t omega; |r|^2, (rHat, r), sum |rHat_i r_i|
    tot[0] = tot[1] = tot[2] = 0.0;
    each([&](int q, uint32_t lc, uint32_t c) {
      const double sv = r[lc];
      double ph = p[lc], sh = sv;
      if (PREC) {
        const double ivc = cells.inverse(A, q, c);
        ph *= ivc;
        sh *= ivc;
      }
      double xv = x_at(lc) + ph * alpha;
      xv = xv + sh * omega;
      set_x(lc, xv);
      const double rn = sv - t[lc] * omega;
      r[lc] = rn;
      const double rhr = rh[lc] * rn;
      tot[0] += rn * rn;
      tot[1] = fma(rh[lc], rn, tot[1]);
      tot[2] += fabs(rhr);
    });
    if (!team.reduce(tot)) return;
    const double res = sqrt(tot[0]);
    rNorm = res;
    if (!isfinite(res)) {
      push(res);
      return finish(CFDB_SOLVER_NONFINITE_RESIDUAL, iter, res);
    }
    completed = iter;
    push(res);
    lastHist = res;
    if (conv(res)) return finish(CFDB_SOLVER_CONVERGED, iter, res);
    rhoOld = rho;
    rho = tot[1];
    rhoTerms = tot[2];
  }
  finish(CFDB_SOLVER_MAX_ITERATIONS, completed, lastHist);
}

}  // namespace res
}  // namespace cfdb
