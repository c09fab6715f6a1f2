// Learned multigrid-shaped preconditioner (see mg.cuh): hierarchy
// construction, the V-cycle kernels, and the FCG(1) solve loop captured as
// one CUDA graph with a device-side WHILE node (the loop runs without a host
// round trip; the last kernel of each iteration decides whether another one
// follows).
//
// Work layout.  Everything runs in kernel space (2D grids as nx x 1 x ny).
// Large levels with rows of whole tiles march in z with four cells per thread
// (mg_quad.cuh), so every array is read from DRAM about once per pass; other
// levels gather, one cell per thread (mg_gather.cuh).  All levels at or below
// 4096 cells run inside ONE thread block with their data in shared memory;
// the levels above them up to 32768 cells, and the whole solve of a small
// system, on one cluster (mg_cluster.cuh).
//
// Reductions are deterministic without a grid barrier: every block stores its
// partial sums, and the last block to finish (atomic ticket) adds all partials
// in block order and publishes the scalars.  Nothing in this file waits on
// another block.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>

#include "cfdb_internal.cuh"
#include "grid_sync.cuh"
#include "mg.cuh"
#include "pcg_internal.cuh"
#include "resident_launch.cuh"

namespace cfdb {

MgWeights mg_default_weights(int dim) {
  MgWeights W;
  std::memset(&W, 0, sizeof(W));
  W.dim = dim;
  W.levels = 1;
  W.nu = 2;
  W.coarse_sweeps = 50;
  for (int l = 0; l < kMgMaxLevels; ++l) {
    W.w[l][13] = 0.8f;  // centre tap: damped Jacobi
    W.c[l] = 1.0f;
  }
  return W;
}

#include "mg_trained.inc"

bool mg_weights_valid(const MgWeights& W, std::string* why) {
  auto fail = [&](const char* m) {
    if (why) *why = m;
    return false;
  };
  if (W.dim != 2 && W.dim != 3) return fail("weights: dim must be 2 or 3");
  if (W.levels < 1 || W.levels > kMgMaxLevels) return fail("weights: levels must be 1..16");
  if (W.nu < 1 || W.nu > 8) return fail("weights: nu must be 1..8");
  if (W.coarse_sweeps < 0 || W.coarse_sweeps > 1000) return fail("weights: coarse sweeps 0..1000");
  for (int l = 0; l < W.levels; ++l) {
    if (!std::isfinite(W.c[l])) return fail("weights: non-finite coarse weight");
    for (int t = 0; t < kMgTaps; ++t) {
      if (!std::isfinite(W.w[l][t])) return fail("weights: non-finite kernel tap");
      if (W.w[l][t] != W.w[l][kMgTaps - 1 - t]) return fail("weights: kernels must be point-symmetric");
      if (W.dim == 2 && (t < 9 || t >= 18) && W.w[l][t] != 0.f)
        return fail("weights: 2D kernels use the middle 3x3 plane only");
    }
  }
  return true;
}

MgHierarchy::~MgHierarchy() {
  for (void* p : owned) cudaFree(p);
}

namespace {

constexpr int kT = 256;                 // threads of the tiled kernels
constexpr int kGridCap = 148 * 8;       // their blocks (8 x 256 threads resident per SM)
constexpr int kMaxBlocks = 148 * 16;    // widest reduction launch
constexpr int64_t kCoarseCells = 4096;
constexpr int kMaxCoarse = 8;
constexpr int kCoarseThreads = 1024;
constexpr size_t kCoarseSmemCap = 200 * 1024;

// Kernels of the solve body are launched with programmatic dependent launch
// allowed: each one waits (griddepcontrol.wait) for its predecessor's
// results before it reads anything, so the launch of a kernel is prepared
// while its predecessor finishes.  (Letting successors start at the top of
// each kernel, launch_dependents, was measured 1-3 % slower: their waiting
// blocks hold resources.)  The wait is a no-op for a kernel launched
// without the attribute.
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// 16-, 8- and 4-byte asynchronous global -> shared copies (cp.async); a copy
// whose source lies outside the level fills its bytes with zeros and reads
// nothing.
__device__ __forceinline__ void cp16(void* dst, const void* src, bool in) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(src), "r"(in ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp8(void* dst, const void* src, bool in) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(src), "r"(in ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void cp4(void* dst, const void* src, bool in) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(s), "l"(src), "r"(in ? 4 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Thread layout of the initial residual's tiles: TX x TY threads, one cell of
// a plane each.
template <int DIM>
struct Tile;
// Shared-memory rows of a plane buffer: the TY rows plus a y-halo row on
// each side when TY > 1 (a 2D row has no y-neighbours).
template <int TY>
struct Rows {
  static constexpr int R0 = TY > 1 ? 1 : 0, N = TY + 2 * R0;
};
template <>
struct Tile<2> {
  static constexpr int TX = 256, TY = 1;
};
template <>
struct Tile<3> {
  static constexpr int TX = 32, TY = 8;
};

struct Kern {
  float w[kMgTaps];  // kernel-space taps: (dk+1)*9 + (dj+1)*3 + (di+1)
};

struct LV {
  int nx, ny, nz;
  const float* fx;
  const float* fy;  // null in 2D
  const float* fz;
  const float* isq;
};

__host__ __device__ inline LV lv(const MgLevel& M) {
  return LV{M.n[0], M.n[1], M.n[2], M.f[0], M.f[1], M.f[2], M.isq};
}

// Level-l kernel in kernel space.  A 2D weight set holds its 3x3 taps in the
// middle plane of the 27 (real (dj, di)); kernel space maps real y to z.
Kern kern_of(const MgWeights& W, int l) {
  const float* w = W.w[std::min(l, W.levels - 1)];
  Kern K;
  if (W.dim == 3) {
    std::memcpy(K.w, w, sizeof(K.w));
  } else {
    std::memset(K.w, 0, sizeof(K.w));
    for (int dj = 0; dj < 3; ++dj)
      for (int di = 0; di < 3; ++di) K.w[dj * 9 + 3 + di] = w[9 + dj * 3 + di];
  }
  return K;
}
float cw_of(const MgWeights& W, int l) { return W.c[std::min(l, W.levels - 1)]; }

}  // namespace

void mg_kernel_taps(const MgWeights& W, int l, float out[kMgTaps]) {
  const Kern K = kern_of(W, l);
  std::memcpy(out, K.w, sizeof(K.w));
}

namespace {

__device__ __forceinline__ int64_t at(const LV& L, int i, int j, int k) {
  return i + (int64_t)L.nx * (j + (int64_t)L.ny * k);
}

struct C7 {
  float xl, xh, yl, yh, zl, zh, d;
};

// Face couplings of cell (i,j,k); boundary faces enter the diagonal only
// (their neighbour values are 0 in every caller).
template <int DIM>
__device__ __forceinline__ C7 coef(const LV& L, int i, int j, int k) {
  C7 c;
  const int64_t bx = i + (int64_t)(L.nx + 1) * (j + (int64_t)L.ny * k);
  c.xl = L.fx[bx];
  c.xh = L.fx[bx + 1];
  if (DIM == 3) {
    const int64_t by = i + (int64_t)L.nx * (j + (int64_t)(L.ny + 1) * k);
    c.yl = L.fy[by];
    c.yh = L.fy[by + L.nx];
  } else {
    c.yl = c.yh = 0.f;
  }
  const int64_t bz = at(L, i, j, k);
  c.zl = L.fz[bz];
  c.zh = L.fz[bz + (int64_t)L.nx * L.ny];
  c.d = ((c.xl + c.xh) + (c.yl + c.yh)) + (c.zl + c.zh);
  return c;
}

__device__ __forceinline__ float apply7(const C7& c, float v, float w, float e, float s, float n,
                                        float b, float t) {
  return c.d * v - (((c.xl * w + c.xh * e) + (c.yl * s + c.yh * n)) + (c.zl * b + c.zh * t));
}

// Parent (coarse) cell of fine cell (i,j,k).
__device__ __forceinline__ int64_t parent(const LV& C, int i, int j, int k) {
  return (i >> 1) + (int64_t)C.nx * ((j >> 1) + (int64_t)C.ny * (k >> 1));
}

// ------------------------------------------------------- tiled plane march

// Work of a tiled pass: tiles x plane pairs; block b takes a contiguous run
// of pair items, so its plane runs start on even planes.
struct Seg {
  int tiles_x;
  int pairs;
  int64_t items;
};

template <int DIM>
Seg make_seg(int nx, int ny, int nz) {
  constexpr int PX = Tile<DIM>::TX, PY = Tile<DIM>::TY;
  Seg s;
  s.tiles_x = (nx + PX - 1) / PX;
  const int64_t tiles = (int64_t)s.tiles_x * ((ny + PY - 1) / PY);
  s.pairs = (nz + 1) / 2;
  s.items = tiles * s.pairs;
  return s;
}

// Blocks for a pass: at most kGridCap, each with the same number of items.
int seg_grid(const Seg& s) {
  const int64_t per = std::max<int64_t>(1, (s.items + kGridCap - 1) / kGridCap);
  return (int)std::max<int64_t>(1, (s.items + per - 1) / per);
}

// f(tix, tiy, k0, k1) for every plane run of this block.
template <class F>
__device__ __forceinline__ void for_runs(const Seg& sg, int nz, F f) {
  const int64_t w0 = sg.items * blockIdx.x / gridDim.x;
  const int64_t w1 = sg.items * (blockIdx.x + 1) / gridDim.x;
  int64_t w = w0;
  while (w < w1) {
    const int64_t tile = w / sg.pairs;
    const int kp0 = (int)(w % sg.pairs);
    const int kp1 = (int)min((int64_t)sg.pairs, kp0 + (w1 - w));
    f((int)(tile % sg.tiles_x), (int)(tile / sg.tiles_x), 2 * kp0, min(nz, 2 * kp1));
    w += kp1 - kp0;
  }
}

// 7-point march over planes [k0, k1) of tile (tix, tiy): val(i,j,k) is the
// stencil input.  For every plane, cell(i, j, k, v, w, e, s, n, b, t) runs for
// the thread's cell if it is in the grid.  z-neighbours stay in registers; the
// plane with its x/y halo is staged in shared memory.
template <typename T, int TX, int TY, class Val, class Cell>
__device__ __forceinline__ void march7(int nx, int ny, int nz, int tix, int tiy, int k0, int k1,
                                       T (*buf)[Rows<TY>::N][TX + 2], Val val, Cell cell) {
  constexpr int R0 = Rows<TY>::R0;
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;
  const int x0 = tix * TX, i = x0 + tx, j = tiy * TY + ty;
  const bool row = j < ny, act = row && i < nx;
  T vp = (act && k0 > 0) ? val(i, j, k0 - 1) : T(0);
  T vc = act ? val(i, j, k0) : T(0);
  for (int k = k0; k < k1; ++k) {
    T(*s)[TX + 2] = buf[k & 1];
    const T vn = (act && k + 1 < nz) ? val(i, j, k + 1) : T(0);
    s[ty + R0][1 + tx] = vc;
    if (tx == 0) s[ty + R0][0] = (row && x0 > 0) ? val(x0 - 1, j, k) : T(0);
    if (tx == TX - 1) s[ty + R0][TX + 1] = (row && x0 + TX < nx) ? val(x0 + TX, j, k) : T(0);
    if (TY > 1) {
      if (ty == 0) s[0][1 + tx] = (j > 0 && i < nx) ? val(i, j - 1, k) : T(0);
      if (ty == TY - 1) s[TY + 1][1 + tx] = (j + 1 < ny && i < nx) ? val(i, j + 1, k) : T(0);
    }
    __syncthreads();
    if (act) {
      const T south = (TY > 1) ? s[ty][1 + tx] : T(0), north = (TY > 1) ? s[ty + 2][1 + tx] : T(0);
      cell(i, j, k, vc, s[ty + R0][tx], s[ty + R0][tx + 2], south, north, vp, vn);
    }
    vp = vc;
    vc = vn;
  }
  __syncthreads();
}

// ----------------------------------------------------------------- FCG state

struct FcgState {
  // set by the host before each solve
  const double* b;
  double* x;
  double abs_tol, rel_tol;
  long long max_it, window;
  // progress
  double b0, res, best;
  double pq, pr, alpha, beta;
  double alpha_prev;  // of the last even iteration, whose x update waits (deferred form)
  long long it, best_it;
  int status, done;
  unsigned ticket;
};

constexpr int kRunning = -1;

// Block partials -> fixed-order total in the last block; fin(tot) runs in
// thread 0 of that block.  Every thread of the block must call this.
template <int NV, bool WIDE = true, class Fin>
__device__ __forceinline__ void reduce_last(double (&v)[NV], double* partials, unsigned* ticket,
                                            Fin fin) {
  __shared__ double red[32 * NV];
  __shared__ int is_last;
  block_sum<NV>(v, red);
  const int nb = gridDim.x * gridDim.y;
  const int b = blockIdx.x + gridDim.x * blockIdx.y;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < NV; ++q) partials[(size_t)b * NV + q] = v[q];
    __threadfence();
    is_last = (atomicAdd(ticket, 1u) == (unsigned)(nb - 1));
  }
  __syncthreads();
  if (is_last) {
    __threadfence();
    double tot[NV];
    if constexpr (WIDE) {
      // every thread of the block takes a strided share of the partials: one
      // warp alone spends several trips to L2 on the 1 000-2 400 of a wide
      // pass (an FCG iteration of 100x75x61 134 -> 128 us; blocks of 64
      // threads gain nothing)
#pragma unroll
      for (int q = 0; q < NV; ++q) tot[q] = 0.0;
#pragma unroll 4
      for (int p = threadIdx.x; p < nb; p += blockDim.x)
#pragma unroll
        for (int q = 0; q < NV; ++q) tot[q] += __ldcg(partials + (size_t)p * NV + q);
      block_sum<NV>(tot, red);
    } else {
      grid_total<NV>(partials, NV, nb, tot, red);
    }
    if (threadIdx.x == 0) {
      fin(tot);
      atomicExch(ticket, 0u);
    }
  }
}

// The WHILE node's condition, or nothing when the kernels run outside a
// graph (stream mode: active = 0).
struct Loop {
  cudaGraphConditionalHandle h;
  int active;
};

__device__ __forceinline__ void set_loop(const Loop& lp, unsigned v) {
  if (lp.active) cudaGraphSetConditional(lp.h, v);
}

__device__ __forceinline__ void stop_loop(FcgState* S, const Loop& h, int status) {
  S->status = status;
  S->done = 1;
  set_loop(h, 0);
}

struct Hook {
  const double* q;  // previous A p
  double* partials;
  FcgState* S;
  Loop h;
};

// ------------------------------------------------------------ level kernels

enum { SM_FIRST = 0, SM_ADD = 1 };

#ifndef CFDB_PDL
#define CFDB_PDL 1
#endif

// The first launch error on this host thread since the last take_launch_error()
// (a launch refused inside a stream capture leaves no node; the capture then
// reports it instead of instantiating an incomplete graph).
thread_local cudaError_t g_launch_error = cudaSuccess;

cudaError_t take_launch_error() {
  const cudaError_t e = g_launch_error;
  g_launch_error = cudaSuccess;
  return e;
}

template <typename... KArgs, typename... Args>
void launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
            Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = CFDB_PDL;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
  if (e != cudaSuccess && g_launch_error == cudaSuccess) g_launch_error = e;
}

// ----------------------------------------------------- coarse-level block

struct CoarseLevel {
  int n[3];
  int cells;
  const float* f[3];  // global sources (f[1] null in 2D)
  const float* isq;
  float* x_glob;      // global x (written back for the first coarse level)
  const float* r_glob;
  int off[7];         // shared-memory offsets (floats): fx fy fz isq x r u
  res::FastDiv dx, dy;
  int warps;          // warps that work on the level
};

struct CoarsePlan {
  int count;
  int nu, sweeps;
  CoarseLevel lv[kMaxCoarse];
  Kern K[kMaxCoarse];
  float cw[kMaxCoarse];
};

// Cells of a padded shared-memory vector (x, res): one zero cell past each
// end of every active axis, so stencil and kernel taps need no bounds tests.
__host__ __device__ inline int coarse_padded(int dim, const int n[3]) {
  return (n[0] + 2) * (dim == 3 ? n[1] + 2 : 1) * (n[2] + 2);
}

// A coarse level as the block sees it: couplings and scales unpadded (global
// order), x and res padded with pitches px (y) and pz (z).
template <int DIM>
struct CoarseGeo {
  int nx, ny, nz, px, pz;
  const float *fx, *fy, *fz, *isq;
  __device__ __forceinline__ int pad(int i, int j, int k) const {
    return (i + 1) + (DIM == 3 ? px * (j + 1) : 0) + pz * (k + 1);
  }
};

// (A x)(c) of a padded x at pc; cell c = i + nx * rest, rest = j + ny * k.
// The arithmetic is coef() / apply7() of the grid kernels, with the x, y and
// z couplings read at x faces c + rest, y faces c + nx k and z faces c.
template <int DIM>
__device__ __forceinline__ float coarse_lap(const CoarseGeo<DIM>& G, int c, int rest, int k, int pc,
                                            const float* x) {
  C7 co;
  co.xl = G.fx[c + rest];
  co.xh = G.fx[c + rest + 1];
  if (DIM == 3) {
    co.yl = G.fy[c + G.nx * k];
    co.yh = G.fy[c + G.nx * k + G.nx];
  } else {
    co.yl = co.yh = 0.f;
  }
  co.zl = G.fz[c];
  co.zh = G.fz[c + G.nx * G.ny];
  co.d = ((co.xl + co.xh) + (co.yl + co.yh)) + (co.zl + co.zh);
  const float s = DIM == 3 ? x[pc - G.px] : 0.f, n = DIM == 3 ? x[pc + G.px] : 0.f;
  return apply7(co, x[pc], x[pc - 1], x[pc + 1], s, n, x[pc - G.pz], x[pc + G.pz]);
}

// sum_o K[o] u(pc + o) over a padded u, taps in (dz, dy, dx) order; a tap
// in the halo adds K[o] * 0.
template <int DIM>
__device__ __forceinline__ float coarse_conv(const CoarseGeo<DIM>& G, const Kern& K, int pc,
                                             const float* u) {
  float s = 0.f;
#pragma unroll
  for (int dk = -1; dk <= 1; ++dk) {
#pragma unroll
    for (int dj = (DIM == 2 ? 0 : -1); dj <= (DIM == 2 ? 0 : 1); ++dj) {
      const float* row = u + pc + dk * G.pz + dj * G.px;
#pragma unroll
      for (int di = -1; di <= 1; ++di) s += K.w[(dk + 1) * 9 + (dj + 1) * 3 + (di + 1)] * row[di];
    }
  }
  return s;
}

// The block-resident tail of the V-cycle: levels cf.. with their couplings,
// scales and vectors in shared memory (the couplings, scales and the first
// level's residual brought in by cp.async, 16 bytes a copy).  Same layers as
// the grid kernels; the first smoothing's scaled residual isq r is formed
// once per cell instead of once per tap, x and res carry a zero halo, and
// all indexing is 32-bit: the kernel runs on one SM and is bound by its
// instruction issue.  Cell coordinates come from FastDiv; every level is worked
// on by only the warps that own its cells (coarse_cycle).

// Zeroes the padded vectors (their halos stay zero).
template <int DIM>
__device__ __forceinline__ void coarse_clear(const CoarsePlan& P, float* sm) {
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int l = 0; l < P.count; ++l) {
    const CoarseLevel& c = P.lv[l];
    const int words = (coarse_padded(DIM, c.n) + 3) >> 2;
    float4* x4 = reinterpret_cast<float4*>(sm + c.off[4]);
    float4* r4 = reinterpret_cast<float4*>(sm + c.off[6]);
    for (int q = tid; q < words; q += nt) {
      x4[q] = make_float4(0.f, 0.f, 0.f, 0.f);
      r4[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
}

// 16-byte copies over the body of an array (every source is its own
// allocation, every destination 16-byte aligned), 4-byte ones for the tail
__device__ __forceinline__ void coarse_fetch(float* dst, const float* src, int count) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const int body = count & ~3;
  for (int q = 4 * tid; q < body; q += 4 * nt) cp16(dst + q, src + q, true);
  for (int q = body + tid; q < count; q += nt) cp4(dst + q, src + q, true);
}

// Issues the copies of every level's couplings and scales.
template <int DIM>
__device__ __forceinline__ void coarse_fetch_levels(const CoarsePlan& P, float* sm) {
  for (int l = 0; l < P.count; ++l) {
    const CoarseLevel& c = P.lv[l];
    coarse_fetch(sm + c.off[0], c.f[0], (c.n[0] + 1) * c.n[1] * c.n[2]);
    if (DIM == 3) coarse_fetch(sm + c.off[1], c.f[1], c.n[0] * (c.n[1] + 1) * c.n[2]);
    coarse_fetch(sm + c.off[2], c.f[2], c.n[0] * c.n[1] * (c.n[2] + 1));
    coarse_fetch(sm + c.off[3], c.isq, c.cells);
  }
}

// One cycle over the levels in shared memory: the first level's r is in
// place; the first level's x (padded) is the result.
//
// The cycle is a chain of some 30 short phases, so what counts is the latency
// of each: a level is worked on by only the warps that own its cells, behind
// a named barrier of its own (the others wait where they are needed again),
// the scaled residual u is formed where r is, and prolongation and Jacobi
// sweeps need no phase of their own (x + c P e is formed as it is read, the
// sweeps alternate between two vectors).  With it a 24^3 FCG iteration took
// 37 us instead of 41, 12^3 21 instead of 26.
template <int DIM>
__device__ __forceinline__ void coarse_cycle(const CoarsePlan& P, float* sm) {
  const int tid = threadIdx.x, warp = tid >> 5;
  const int last = P.count - 1;
  // a level as this thread works on it, in registers: its geometry, vectors
  // and the thread's first cell (on the smaller levels its only one)
  struct Cell {
    int i, j, k, c, rest, pc;
  };
  struct Level : CoarseGeo<DIM> {
    int cells, nt, id;
    res::FastDiv dx, dy;
    float *x, *r, *u;
    Cell first;
    __device__ __forceinline__ Cell cell(int c) const {
      Cell o;
      o.c = c;
      o.rest = (int)dx.div((uint32_t)c);
      o.i = c - o.rest * this->nx;
      o.k = DIM == 3 ? (int)dy.div((uint32_t)o.rest) : o.rest;
      o.j = DIM == 3 ? o.rest - o.k * this->ny : 0;
      o.pc = this->pad(o.i, o.j, o.k);
      return o;
    }
    __device__ __forceinline__ void sync() const {
      asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nt) : "memory");
    }
  };
  auto geo = [&](int l) {
    const CoarseLevel& c = P.lv[l];
    Level G;
    G.nx = c.n[0];
    G.ny = c.n[1];
    G.nz = c.n[2];
    G.px = c.n[0] + 2;
    G.pz = DIM == 3 ? G.px * (c.n[1] + 2) : G.px;
    G.fx = sm + c.off[0];
    G.fy = DIM == 3 ? sm + c.off[1] : nullptr;
    G.fz = sm + c.off[2];
    G.isq = sm + c.off[3];
    G.x = sm + c.off[4];
    G.r = sm + c.off[5];
    G.u = sm + c.off[6];
    G.cells = c.cells;
    G.nt = 32 * c.warps;
    G.id = l + 1;
    G.dx = c.dx;
    G.dy = c.dy;
    G.first = G.cell(tid);
    return G;
  };
  // f(cell) for every cell of a level, by its warps
  auto cells_of = [&](const Level& G, auto f) {
    if (tid < G.cells) f(G.first);
    for (int c = tid + G.nt; c < G.cells; c += G.nt) f(G.cell(c));
  };
  auto mine = [&](int l) { return warp < P.lv[l].warps; };
  // u = D^-1/2 r, or x after the first of the coarsest level's sweeps
  const int sweeps = P.sweeps, nu = P.nu;
  auto start = [&](int l, const Level& G, const Cell& q, float r) {
    const float is = G.isq[q.c];
    if (l < last) G.u[q.pc] = is * r;
    else G.x[q.pc] = sweeps > 0 ? 0.8f * (is * is) * r : 0.f;
  };
  auto lap = [&](const Level& G, const Cell& q, const float* x) {
    return coarse_lap<DIM>(G, q.c, q.rest, q.k, q.pc, x);
  };
  if (mine(0)) {
    const Level G = geo(0);
    cells_of(G, [&](const Cell& q) { start(0, G, q, G.r[q.c]); });
    G.sync();
  }
  int deepest = -1;  // the last level this warp works on
  for (int l = 0; l < last; ++l) {
    if (!mine(l)) break;
    deepest = l;
    const Level G = geo(l);
    const Kern& K = P.K[l];
    cells_of(G, [&](const Cell& q) { G.x[q.pc] = G.isq[q.c] * coarse_conv<DIM>(G, K, q.pc, G.u); });
    G.sync();
    for (int s = 1; s < nu; ++s) {
      cells_of(G, [&](const Cell& q) { G.u[q.pc] = G.isq[q.c] * (G.r[q.c] - lap(G, q, G.x)); });
      G.sync();
      cells_of(G, [&](const Cell& q) { G.x[q.pc] += G.isq[q.c] * coarse_conv<DIM>(G, K, q.pc, G.u); });
      G.sync();
    }
    cells_of(G, [&](const Cell& q) { G.u[q.pc] = G.r[q.c] - lap(G, q, G.x); });
    G.sync();
    if (!mine(l + 1)) break;
    // restriction: the sum over the 2 x 2 (x 2) children, (z, y, x) order;
    // children past an odd edge are halo zeros
    const Level C = geo(l + 1);
    cells_of(C, [&](const Cell& q) {
      float s = 0.f;
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < (DIM == 3 ? 2 : 1); ++b)
#pragma unroll
          for (int t = 0; t < 2; ++t) s += G.u[G.pad(2 * q.i + t, 2 * q.j + b, 2 * q.k + a)];
      C.r[q.c] = s;
      start(l + 1, C, q, s);
    });
    C.sync();
    deepest = l + 1;
  }
  if (mine(last)) {
    deepest = last;
    const Level G = geo(last);
    float *x = G.x, *y = G.u;
    for (int s = 1; s < sweeps; ++s) {
      cells_of(G, [&](const Cell& q) {
        const float is = G.isq[q.c];
        y[q.pc] = x[q.pc] + 0.8f * (is * is) * (G.r[q.c] - lap(G, q, x));
      });
      G.sync();
      float* t = x;
      x = y;
      y = t;
    }
    if (x != G.x) {  // the result belongs in x
      cells_of(G, [&](const Cell& q) { y[q.pc] = x[q.pc]; });
      if (last == 0) G.sync();
    }
  }
  for (int l = min(last - 1, deepest); l >= 0; --l) {
    const Level G = geo(l);
    const CoarseLevel& cl = P.lv[l + 1];
    const int cpx = cl.n[0] + 2, cpz = DIM == 3 ? cpx * (cl.n[1] + 2) : cpx;
    const float* ec = sm + cl.off[4];
    const Kern& K = P.K[l];
    const float cw = P.cw[l];
    // c P e at a cell, 0 outside the domain (x's own halo is 0)
    auto e = [&](int i, int j, int k) {
      const float v = ec[((i >> 1) + 1) + (DIM == 3 ? cpx * ((j >> 1) + 1) : 0) + cpz * ((k >> 1) + 1)];
      const bool in = i >= 0 && i < G.nx && k >= 0 && k < G.nz && (DIM == 2 || (j >= 0 && j < G.ny));
      return in ? cw * v : 0.f;
    };
    G.sync();  // the level below is done (its warps are among this level's)
    for (int s = 0; s < nu; ++s) {
      cells_of(G, [&](const Cell& q) {
        float ax;
        if (s == 0) {
          C7 co;
          co.xl = G.fx[q.c + q.rest];
          co.xh = G.fx[q.c + q.rest + 1];
          co.yl = DIM == 3 ? G.fy[q.c + G.nx * q.k] : 0.f;
          co.yh = DIM == 3 ? G.fy[q.c + G.nx * q.k + G.nx] : 0.f;
          co.zl = G.fz[q.c];
          co.zh = G.fz[q.c + G.nx * G.ny];
          co.d = ((co.xl + co.xh) + (co.yl + co.yh)) + (co.zl + co.zh);
          const float* x = G.x + q.pc;
          ax = apply7(co, x[0] + e(q.i, q.j, q.k), x[-1] + e(q.i - 1, q.j, q.k),
                      x[1] + e(q.i + 1, q.j, q.k), DIM == 3 ? x[-G.px] + e(q.i, q.j - 1, q.k) : 0.f,
                      DIM == 3 ? x[G.px] + e(q.i, q.j + 1, q.k) : 0.f, x[-G.pz] + e(q.i, q.j, q.k - 1),
                      x[G.pz] + e(q.i, q.j, q.k + 1));
        } else {
          ax = lap(G, q, G.x);
        }
        G.u[q.pc] = G.isq[q.c] * (G.r[q.c] - ax);
      });
      G.sync();
      cells_of(G, [&](const Cell& q) {
        float v = G.x[q.pc] + G.isq[q.c] * coarse_conv<DIM>(G, K, q.pc, G.u);
        if (s == 0) v += e(q.i, q.j, q.k);
        G.x[q.pc] = v;
      });
      if (s + 1 < nu) G.sync();
    }
  }
  __syncthreads();
}

// A plan's copy in shared memory (T: a multiple of 4 bytes), whose levels are
// indexed at run time: an indexed read of a kernel parameter goes through
// the constant cache, which these plans (3 KB, read by every warp) thrash.
template <class T>
__device__ __forceinline__ const T& to_shared(const T& src, void* dst) {
  static_assert(sizeof(T) % 4 == 0, "whole words");
  const unsigned* s = reinterpret_cast<const unsigned*>(&src);
  unsigned* d = reinterpret_cast<unsigned*>(dst);
  for (int q = threadIdx.x; q < (int)(sizeof(T) / 4); q += blockDim.x) d[q] = s[q];
  __syncthreads();
  return *reinterpret_cast<const T*>(dst);
}
// Floats a plan's copy takes at the front of dynamic shared memory.
template <class T>
constexpr int plan_words() {
  return (int)((sizeof(T) + 15) / 16) * 4;
}

template <int DIM>
__global__ void __launch_bounds__(kCoarseThreads) k_coarse(const __grid_constant__ CoarsePlan arg) {
  extern __shared__ float4 smem4[];
  const CoarsePlan& P = to_shared(arg, smem4);
  float* sm = reinterpret_cast<float*>(smem4) + plan_words<CoarsePlan>();
  coarse_clear<DIM>(P, sm);
  pdl_enter();
  coarse_fetch_levels<DIM>(P, sm);
  coarse_fetch(sm + P.lv[0].off[5], P.lv[0].r_glob, P.lv[0].cells);
  cp_commit();
  cp_wait<0>();
  __syncthreads();
  coarse_cycle<DIM>(P, sm);
  const CoarseLevel& c0 = P.lv[0];
  const float* x0 = sm + c0.off[4];
  const int px = c0.n[0] + 2, pz = DIM == 3 ? px * (c0.n[1] + 2) : px;
  const float inx = 1.0f / (float)c0.n[0], iny = 1.0f / (float)c0.n[1];
  for (int c = threadIdx.x; c < c0.cells; c += blockDim.x) {
    const int rest = __float2int_rz(((float)c + 0.5f) * inx);
    const int k = DIM == 3 ? __float2int_rz(((float)rest + 0.5f) * iny) : rest;
    const int j = DIM == 3 ? rest - k * c0.n[1] : 0;
    c0.x_glob[c] = x0[(c - rest * c0.n[0] + 1) + (DIM == 3 ? px * (j + 1) : 0) + pz * (k + 1)];
  }
}

// ------------------------------------------------------ hierarchy build

__global__ void k_faces0(float* out, int e0, int e1, int e2, int axis, const double* full,
                         const double* table) {
  const int64_t m = (int64_t)e0 * e1 * e2;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < m;
       q += (int64_t)gridDim.x * blockDim.x) {
    double v;
    if (full) {
      v = full[q];
    } else {
      const int i = (int)(q % e0);
      const int64_t rest = q / e0;
      const int j = (int)(rest % e1), k = (int)(rest / e1);
      v = table[axis == 0 ? i : (axis == 1 ? j : k)];
    }
    out[q] = (float)v;
  }
}

// Coarse faces of axis a: sum of the fine faces they cover.
__global__ void k_agglomerate(MgLevel F, MgLevel C, int a) {
  int ext[3] = {C.n[0], C.n[1], C.n[2]};
  ext[a] += 1;
  int fext[3] = {F.n[0], F.n[1], F.n[2]};
  fext[a] += 1;
  const int64_t m = (int64_t)ext[0] * ext[1] * ext[2];
  const int b1 = (a == 0) ? 1 : 0, b2 = (a == 2) ? 1 : 2;
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < m;
       q += (int64_t)gridDim.x * blockDim.x) {
    int cc[3];
    cc[0] = (int)(q % ext[0]);
    const int64_t rest = q / ext[0];
    cc[1] = (int)(rest % ext[1]);
    cc[2] = (int)(rest / ext[1]);
    const int fa = (cc[a] == C.n[a]) ? F.n[a] : 2 * cc[a];
    float s = 0.f;
    for (int u = 0; u < 2; ++u)
      for (int v = 0; v < 2; ++v) {
        int fc[3];
        fc[a] = fa;
        fc[b1] = 2 * cc[b1] + u;
        fc[b2] = 2 * cc[b2] + v;
        if (fc[b1] >= F.n[b1] || fc[b2] >= F.n[b2]) continue;
        s += F.f[a][fc[0] + (int64_t)fext[0] * (fc[1] + (int64_t)fext[1] * fc[2])];
      }
    C.f[a][q] = s;
  }
}

template <int DIM>
__global__ void k_isq(MgLevel M) {
  const LV L = lv(M);
  for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < M.cells;
       q += (int64_t)gridDim.x * blockDim.x) {
    const int i = (int)(q % L.nx);
    const int64_t rest = q / L.nx;
    const int j = (int)(rest % L.ny), k = (int)(rest / L.ny);
    const float d = coef<DIM>(L, i, j, k).d;
    M.isq[q] = d > 0.f ? rsqrtf(d) : 0.f;
  }
}

int flat_grid(int64_t n) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, kMaxBlocks));
}

bool axis_active(int dim, int a) { return dim == 3 || a != 1; }

cfdb_status refresh_values(cfdb_context* ctx, MgHierarchy& H, const FineOperator& op) {
  cudaStream_t st = ctx->stream;
  int launches = 0;
  for (int l = 0; l < H.levels; ++l) {
    MgLevel& M = H.L[l];
    for (int a = 0; a < 3; ++a) {
      if (!axis_active(H.dim, a)) continue;
      int e[3] = {M.n[0], M.n[1], M.n[2]};
      e[a] += 1;
      const int64_t m = (int64_t)e[0] * e[1] * e[2];
      if (l == 0)
        k_faces0<<<flat_grid(m), 256, 0, st>>>(M.f[a], e[0], e[1], e[2], a, op.full[a], op.table[a]);
      else
        k_agglomerate<<<flat_grid(m), 256, 0, st>>>(H.L[l - 1], M, a);
      ++launches;
    }
    if (H.dim == 2) k_isq<2><<<flat_grid(M.cells), 256, 0, st>>>(M);
    else k_isq<3><<<flat_grid(M.cells), 256, 0, st>>>(M);
    ++launches;
  }
  CFDB_CHECK_LAUNCH(ctx);
  count_launch(ctx, launches);
  return CFDB_OK;
}

// --------------------------------------------------------- cycle enqueue

size_t up4(int64_t n) { return (size_t)((n + 3) & ~(int64_t)3); }

size_t coarse_bytes(const MgHierarchy& H, int from) {
  size_t floats = 0;
  for (int l = from; l < H.levels; ++l) {
    const MgLevel& M = H.L[l];
    floats += up4((int64_t)(M.n[0] + 1) * M.n[1] * M.n[2]) + up4((int64_t)M.n[0] * M.n[1] * (M.n[2] + 1));
    if (H.dim == 3) floats += up4((int64_t)M.n[0] * (M.n[1] + 1) * M.n[2]);
    floats += 2 * up4(M.cells) + 2 * up4(coarse_padded(H.dim, M.n));
  }
  return floats * sizeof(float);
}

// The levels [from, ...) in one block of `threads`.
CoarsePlan coarse_plan(const MgHierarchy& H, const MgWeights& W, int from, int threads) {
  CoarsePlan P;
  std::memset(&P, 0, sizeof(P));
  P.count = H.levels - from;
  P.nu = W.nu;
  P.sweeps = W.coarse_sweeps;
  int off = 0;
  auto take = [&](int64_t n) {
    const int o = off;
    off += (int)up4(n);  // 16-byte aligned sub-arrays
    return o;
  };
  for (int q = 0; q < P.count; ++q) {
    const MgLevel& M = H.L[from + q];
    CoarseLevel& c = P.lv[q];
    for (int a = 0; a < 3; ++a) c.n[a] = M.n[a];
    c.cells = (int)M.cells;
    for (int a = 0; a < 3; ++a) c.f[a] = M.f[a];
    c.isq = M.isq;
    c.x_glob = M.x;
    c.r_glob = M.r;
    c.off[0] = take((int64_t)(c.n[0] + 1) * c.n[1] * c.n[2]);
    c.off[1] = H.dim == 3 ? take((int64_t)c.n[0] * (c.n[1] + 1) * c.n[2]) : 0;
    c.off[2] = take((int64_t)c.n[0] * c.n[1] * (c.n[2] + 1));
    c.off[3] = take(c.cells);                          // isq
    c.off[4] = take(coarse_padded(H.dim, c.n));        // x (padded)
    c.off[5] = take(c.cells);                          // r
    c.off[6] = take(coarse_padded(H.dim, c.n));        // u (padded)
    c.dx = res::fast_div(c.n[0]);
    c.dy = res::fast_div(c.n[1]);
    c.warps = std::min(threads / 32, (c.cells + 31) / 32);
    P.K[q] = kern_of(W, from + q);
    P.cw[q] = cw_of(W, from + q);
  }
  return P;
}

// Levels of at most this many cells gather even where the quad kernels could
// take them: a march chains a few dependent load and barrier steps per block
// for almost no data.  FCG iteration (us) with 2^16 / 2^19 / 2^21: 512^2
// 70.0 / 65.7 / 63.5, 1024^2 120 / 112.8 / 117.4, 2048^2 242 / 232.5 / 236,
// 128x100x90 - / 155 / 166, 128^3 199 / 199 / 247.
constexpr int64_t kGatherCells = 1 << 19;
// The 2D direction pass likewise: 300^2 57.0 -> 54.0 us, 512^2 63.5 -> 66.2.
constexpr int64_t kGatherDirCells = 1 << 17;

#include "mg_quad.cuh"
#include "mg_stage.cuh"
#include "mg_gather.cuh"

// Blocks of `fn` resident on the whole current GPU at `threads` threads per
// block and `dyn` bytes of dynamic shared memory (registers and shared
// memory permitting), cached per kernel and device.  A kernel that takes
// dynamic shared memory is opted in to `dyn` bytes on the device's first
// query (without it, static plus dynamic shared memory above 48 KB fails the
// launch).  A quad pass launched with at most this many blocks runs in one
// wave.
int one_wave(const void* fn, int threads, size_t dyn = 0) {
  static std::mutex mu;  // contexts on other host threads share the cache
  static std::map<std::pair<const void*, int>, int> cache;
  std::lock_guard<std::mutex> lock(mu);
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    dev = 0;
  }
  auto it = cache.find({fn, dev});
  if (it != cache.end()) return it->second;
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) {
    cudaGetLastError();
    sms = 148;
  }
  if (dyn > 0) cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
  int per = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, threads, dyn) != cudaSuccess || per < 1) {
    cudaGetLastError();
    per = 1;
  }
  return cache[{fn, dev}] = per * sms;
}

template <int DIM>
int quad_wave(const void* fn, const Seg& sg, size_t dyn = 0) {
  return quad_grid<DIM>(sg, one_wave(fn, Quad<DIM>::TX * Quad<DIM>::TY, dyn));
}

// Answers every quad pass's occupancy query once, before any stream capture.
void warm_quad_waves() {
  const Seg sg{1, 1, 1};
  quad_wave<2>((const void*)k_res_q<2, false, true>, sg);
  quad_wave<2>((const void*)k_res_q<2, true, false>, sg);
  quad_wave<2>((const void*)k_res_q<2, false, false>, sg);
  quad_wave<2>((const void*)k_sm_q<2, SM_FIRST, false>, sg);
  quad_wave<2>((const void*)k_sm_q<2, SM_ADD, true>, sg);
  quad_wave<2>((const void*)k_sm_q<2, SM_ADD, false>, sg);
  quad_wave<3>((const void*)k_res_s<false, true>, sg, res_s_smem());
  quad_wave<3>((const void*)k_res_s<true, false>, sg, res_s_smem());
  quad_wave<3>((const void*)k_res_s<false, false>, sg, res_s_smem());
  quad_wave<3>((const void*)k_sm_s<SM_FIRST, false>, sg, sm_s_smem());
  quad_wave<3>((const void*)k_sm_s<SM_ADD, true>, sg, sm_s_smem());
  quad_wave<3>((const void*)k_sm_s<SM_ADD, false>, sg, sm_s_smem());
  quad_wave<3>((const void*)k_dir_s<true>, sg, dir_s_smem());
  quad_wave<3>((const void*)k_dir_s<false>, sg, dir_s_smem());
}

// Whether a level's passes gather (mg_gather.cuh) rather than march in quads.
// Their residual passes leave u = D^-1/2 res for their smoothing passes.
template <int DIM>
bool gathers(const MgLevel& M) {
  return !quad_ok<DIM>(M.n[0]) || M.cells <= kGatherCells;
}
GLevel gcoarse(const LV& C) {
  GLevel G;
  G.L = C;
  G.dx = res::fast_div(C.nx);
  G.dy = res::fast_div(C.ny);
  G.n = (uint32_t)C.nx * C.ny * C.nz;
  return G;
}

template <int DIM>
void level_res(const MgLevel& M, const LV& LC, const float* x, const float* ec, float cw,
               const float* r, float* res, float* rc, int64_t skip, cudaStream_t st) {
  if (gathers<DIM>(M)) {
    const GLevel G = glevel(M);
    const int g = gather_blocks(M.cells);
    if (rc) {
      const GLevel C = gcoarse(LC);
      launch(k_restrict_g<DIM>, gather_blocks(C.n), 256, 0, st, G, C, x, r, rc, (uint32_t)skip);
    } else if (ec) {
      launch(k_resid_g<DIM, true>, g, 256, 0, st, G, LC, x, ec, cw, r, res, (uint32_t)skip);
    } else {
      launch(k_resid_g<DIM, false>, g, 256, 0, st, G, LC, x, ec, cw, r, res, (uint32_t)skip);
    }
  } else if constexpr (DIM == 3) {
    const Seg sg = make_quad_seg<3>(M.n[0], M.n[1], M.n[2]);
    constexpr int T = PlaneTile::T;
    constexpr size_t SM = res_s_smem();
    const LV L = lv(M);
    if (rc)
      launch(k_res_s<false, true>, quad_wave<3>((const void*)k_res_s<false, true>, sg, SM), T, SM,
             st, L, LC, sg, x, ec, cw, r, res, rc, skip);
    else if (ec)
      launch(k_res_s<true, false>, quad_wave<3>((const void*)k_res_s<true, false>, sg, SM), T, SM,
             st, L, LC, sg, x, ec, cw, r, res, rc, skip);
    else
      launch(k_res_s<false, false>, quad_wave<3>((const void*)k_res_s<false, false>, sg, SM), T, SM,
             st, L, LC, sg, x, ec, cw, r, res, rc, skip);
  } else {
    const Seg sg = make_quad_seg<2>(M.n[0], M.n[1], M.n[2]);
    constexpr int T = Quad<2>::TX;
    const LV L = lv(M);
    if (rc)
      launch(k_res_q<2, false, true>, quad_wave<2>((const void*)k_res_q<2, false, true>, sg), T,
             0, st, L, LC, sg, x, ec, cw, r, res, rc, skip);
    else if (ec)
      launch(k_res_q<2, true, false>, quad_wave<2>((const void*)k_res_q<2, true, false>, sg), T,
             0, st, L, LC, sg, x, ec, cw, r, res, rc, skip);
    else
      launch(k_res_q<2, false, false>, quad_wave<2>((const void*)k_res_q<2, false, false>, sg), T,
             0, st, L, LC, sg, x, ec, cw, r, res, rc, skip);
  }
}

template <int DIM>
void level_sm(const MgLevel& M, const LV& LC, const Kern& K, bool first, const float* src,
              const float* ec, float cw, float* x, int64_t skip, int64_t pin, const float* r,
              const Hook* hook, cudaStream_t st) {
  if (gathers<DIM>(M)) {
    const GLevel G = glevel(M);
    const int g = gather_blocks(M.cells);
    if (first)
      launch(k_first_g<DIM>, g, 256, 0, st, G, K, src, x, (uint32_t)skip);
    else if (hook)
      launch(k_smooth_g<DIM, true>, g, 256, 0, st, G, LC, K, src, ec, cw, x, (uint32_t)pin, r, *hook);
    else
      launch(k_smooth_g<DIM, false>, g, 256, 0, st, G, LC, K, src, ec, cw, x, (uint32_t)pin, r, Hook{});
  } else if constexpr (DIM == 3) {
    const Seg sg = make_quad_seg<3>(M.n[0], M.n[1], M.n[2]);
    constexpr int T = PlaneTile::T;
    constexpr size_t SM = sm_s_smem();
    const LV L = lv(M);
    if (first)
      launch(k_sm_s<SM_FIRST, false>, quad_wave<3>((const void*)k_sm_s<SM_FIRST, false>, sg, SM), T,
             SM, st, L, LC, sg, K, src, ec, cw, x, skip, pin, r, Hook{});
    else if (hook)
      launch(k_sm_s<SM_ADD, true>, quad_wave<3>((const void*)k_sm_s<SM_ADD, true>, sg, SM), T, SM, st,
             L, LC, sg, K, src, ec, cw, x, skip, pin, r, *hook);
    else
      launch(k_sm_s<SM_ADD, false>, quad_wave<3>((const void*)k_sm_s<SM_ADD, false>, sg, SM), T, SM,
             st, L, LC, sg, K, src, ec, cw, x, skip, pin, r, Hook{});
  } else {
    const Seg sg = make_quad_seg<2>(M.n[0], M.n[1], M.n[2]);
    constexpr int T = Quad<2>::TX;
    const LV L = lv(M);
    if (first)
      launch(k_sm_q<2, SM_FIRST, false>, quad_wave<2>((const void*)k_sm_q<2, SM_FIRST, false>, sg),
             T, 0, st, L, LC, sg, K, src, ec, cw, x, skip, pin, r, Hook{});
    else if (hook)
      launch(k_sm_q<2, SM_ADD, true>, quad_wave<2>((const void*)k_sm_q<2, SM_ADD, true>, sg), T, 0,
             st, L, LC, sg, K, src, ec, cw, x, skip, pin, r, *hook);
    else
      launch(k_sm_q<2, SM_ADD, false>, quad_wave<2>((const void*)k_sm_q<2, SM_ADD, false>, sg), T,
             0, st, L, LC, sg, K, src, ec, cw, x, skip, pin, r, Hook{});
  }
}

#include "mg_cluster.cuh"

// Levels of at most this many cells (below level 0) run in the cluster's one
// launch instead of four grid kernels each.  An FCG iteration (us, before):
// 300^2 64.4 (72.3), 512^2 74.9 (78.9), 1024^2 125.3 (131.5), 2048^2 250
// (257), 80x48x48 96.0 (101), 100x75x61 134 (142), 256^3 752 (754).
constexpr int64_t kTailCells = 32768;
// Systems of at most this many cells run their whole FCG loop in a cluster
// where it has the shared memory (2D to 256^2, 3D to about 36^3): 129^2 26.6
// us an iteration (graph of grid kernels: 55.8), 256^2 40 (57.6), 12^3 14
// (48), 24^3 29 (62), 33^3 48 (76).
constexpr int64_t kFcgClusterCells = 65536;

// Whether `fn` can run as a cluster of kMaxCluster blocks.
template <class Fn>
bool cluster_ok(Fn fn) {
  return res::cluster_limit((const void*)fn, kClusterT) >= res::kMaxCluster;
}

// First level of the cluster's launch and its layout (words = 0: none).
template <int DIM>
int tail_from(const MgHierarchy& H, const MgWeights& W, ClusterLayout* C) {
  for (int l = 1; l < H.coarse_from && cluster_ok(k_tail<DIM>); ++l) {
    if (H.L[l].cells > kTailCells) continue;
    *C = cluster_layout(H, W, l, false, H.L[l].r, H.L[l].x);
    if (C->words > 0) return l;
  }
  return H.coarse_from;
}

template <typename... KArgs, typename... Args>
void launch_in_cluster(void (*kernel)(KArgs...), size_t smem, cudaStream_t st, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = res::kMaxCluster;
  cfg.blockDim = kClusterT;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = res::kMaxCluster;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = CFDB_PDL;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
  if (e != cudaSuccess && g_launch_error == cudaSuccess) g_launch_error = e;
}

// Enqueues z = M r (level-0 FP32 vectors) on `st`; returns the number of
// kernels launched.
template <int DIM>
int enqueue_cycle(const MgHierarchy& H, const MgWeights& W, const float* r0, float* z0,
                  int64_t skip, const Hook* hook, cudaStream_t st) {
  int launches = 0;
  const int cf = H.coarse_from;
  ClusterLayout CL;
  const int tf = tail_from<DIM>(H, W, &CL);
  auto rp = [&](int l) -> const float* { return l == 0 ? r0 : H.L[l].r; };
  auto xp = [&](int l) -> float* { return l == 0 ? z0 : H.L[l].x; };
  for (int l = 0; l < tf; ++l) {
    const MgLevel& M = H.L[l];
    const LV LC = lv(H.L[l + 1]);
    const Kern K = kern_of(W, l);
    const int64_t sk = l == 0 ? skip : -1;
    level_sm<DIM>(M, LC, K, true, rp(l), nullptr, 0.f, xp(l), sk, -1, nullptr, nullptr, st);
    ++launches;
    for (int q = 1; q < W.nu; ++q) {
      level_res<DIM>(M, LC, xp(l), nullptr, 0.f, rp(l), M.res, nullptr, sk, st);
      level_sm<DIM>(M, LC, K, false, M.res, nullptr, 0.f, xp(l), -1, -1, nullptr, nullptr, st);
      launches += 2;
    }
    level_res<DIM>(M, LC, xp(l), nullptr, 0.f, rp(l), nullptr, H.L[l + 1].r, sk, st);
    ++launches;
  }
  if (tf < cf) {
    launch_in_cluster(k_tail<DIM>, sizeof(float) * (size_t)CL.words, st, CL.P, CL.Q, CL.words);
    ++launches;
  } else if (cf < H.levels) {
    const CoarsePlan P = coarse_plan(H, W, cf, kCoarseThreads);
    launch(k_coarse<DIM>, 1, kCoarseThreads, H.coarse_smem + sizeof(float) * plan_words<CoarsePlan>(), st, P);
    ++launches;
  }
  for (int l = tf - 1; l >= 0; --l) {
    const MgLevel& M = H.L[l];
    const MgLevel& C = H.L[l + 1];
    const LV LC = lv(C);
    const Kern K = kern_of(W, l);
    const float cw = cw_of(W, l);
    const int64_t sk = l == 0 ? skip : -1;
    for (int q = 0; q < W.nu; ++q) {
      const float* ec = q == 0 ? C.x : nullptr;
      level_res<DIM>(M, LC, xp(l), ec, cw, rp(l), M.res, nullptr, sk, st);
      const bool last = (l == 0 && q == W.nu - 1);
      level_sm<DIM>(M, LC, K, false, M.res, ec, cw, xp(l), -1, last ? sk : -1, rp(l),
                    last ? hook : nullptr, st);
      launches += 2;
    }
  }
  return launches;
}

// Algorithmic bytes of one V-cycle: FP32 words read and written per level,
// each array counted once per kernel (faces: about one word per cell and
// active axis).
double cycle_bytes(const MgHierarchy& H, const MgWeights& W) {
  const double d = H.dim, fr = 1.0 / (H.dim == 3 ? 8.0 : 4.0);
  double words = 0.0;
  for (int l = 0; l < H.coarse_from; ++l) {
    const double n = (double)H.L[l].cells;
    const double resid = 3.0 + d, smooth = 4.0;
    const double down = 3.0 + (W.nu - 1) * (resid + smooth) + (2.0 + d + fr);
    const double up = (3.0 + d + fr) + (smooth + fr) + (W.nu - 1) * (resid + smooth);
    words += n * (down + up);
  }
  if (H.coarse_from < H.levels) words += 2.0 * (double)H.L[H.coarse_from].cells;
  return words * 4.0;
}

// ------------------------------------------------------------ FCG kernels

// r = b - A x, r32 = float(r); ||r|| decides whether the loop runs at all.
template <int DIM>
__global__ void __launch_bounds__(kT, 2) k_fcg_init(OpView<double> A, Seg sg, FcgState* S,
                                                    double* __restrict__ r, float* __restrict__ r32,
                                                    double* partials, double* hist, int64_t hcap,
                                                    Loop h) {
  pdl_enter();
  constexpr int TX = Tile<DIM>::TX, TY = Tile<DIM>::TY;
  __shared__ double buf[2][Rows<TY>::N][TX + 2];
  const double* __restrict__ b = S->b;
  const double* __restrict__ x = S->x;
  double acc[1] = {0.0};
  auto val = [&](int i, int j, int k) { return x[i + (int64_t)A.nx * (j + (int64_t)A.ny * k)]; };
  for_runs(sg, A.nz, [&](int tix, int tiy, int k0, int k1) {
    march7<double, TX, TY>(
        A.nx, A.ny, A.nz, tix, tiy, k0, k1, buf, val,
        [&](int i, int j, int k, double v, double w, double e, double s, double n, double bo, double t) {
          const int64_t c = i + (int64_t)A.nx * (j + (int64_t)A.ny * k);
          const double rn = b[c] - apply_coef(load_coef(A, i, j, k), v, w, e, s, n, bo, t);
          r[c] = rn;
          r32[c] = (float)rn;
          acc[0] += rn * rn;
        });
  });
  reduce_last<1>(acc, partials, &S->ticket, [&](const double* tot) {
    const double b0 = sqrt(tot[0]);
    S->b0 = b0;
    S->res = b0;
    S->best = b0;
    S->it = 0;
    S->best_it = 0;
    S->beta = 0.0;
    if (hcap > 0) hist[0] = b0;
    // CG.cpp:49-63: a zero or already converged start returns at once
    if (!isfinite(b0)) {
      stop_loop(S, h, CFDB_SOLVER_NONFINITE_RESIDUAL);
    } else if (b0 == 0.0 || b0 <= S->abs_tol || 1.0 <= S->rel_tol) {
      stop_loop(S, h, CFDB_SOLVER_CONVERGED);
    } else {
      S->status = kRunning;
      S->done = 0;
      set_loop(h, 1);
    }
  });
}

// The update of this thread's cells.  XS: how many directions go into x --
// 1 the current one, 2 the last even iteration's before it, 0 none (it waits).
template <int XS>
__device__ __forceinline__ double fcg_update_cells(int64_t n, double alpha, double alpha_prev,
                                                   double* __restrict__ x, double* __restrict__ r,
                                                   float* __restrict__ r32,
                                                   const double* __restrict__ p,
                                                   const double* __restrict__ pp,
                                                   const double* __restrict__ q) {
  double acc = 0.0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  // four cells per thread in 16-byte vectors, then the remainder one by
  // one; the solver's own arrays start 256-byte aligned, the caller's x may
  // not (then every cell takes the scalar loop)
  const bool vec = (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
  const int64_t n4 = vec ? n / 4 : 0;
  for (int64_t g = tid; g < n4; g += stride) {
    const int64_t c = 4 * g;
    V4<double> xv, pv, ov, rv = ld4(r + c);
    const V4<double> qv = ld4(q + c);
    if (XS >= 1) xv = ld4(x + c), pv = ld4(p + c);
    if (XS >= 2) ov = ld4(pp + c);
    V4<float> rf;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (XS >= 2) xv.v[u] = fma(alpha_prev, ov.v[u], xv.v[u]);
      if (XS >= 1) xv.v[u] = fma(alpha, pv.v[u], xv.v[u]);
      const double rn = fma(-alpha, qv.v[u], rv.v[u]);
      rv.v[u] = rn;
      rf.v[u] = (float)rn;
      acc += rn * rn;
    }
    if (XS >= 1) st4(x + c, xv);
    st4(r + c, rv);
    st4(r32 + c, rf);
  }
  for (int64_t c = 4 * n4 + tid; c < n; c += stride) {
    if (XS >= 2) x[c] = fma(alpha, p[c], fma(alpha_prev, pp[c], x[c]));
    else if (XS >= 1) x[c] = fma(alpha, p[c], x[c]);
    const double rn = fma(-alpha, q[c], r[c]);
    r[c] = rn;
    r32[c] = (float)rn;
    acc += rn * rn;
  }
  return acc;
}

// Systems from this many cells on update x every second iteration, with both
// directions (the double buffer still holds the older one): 8 B a cell and
// iteration less in a pass that streams at the memory's rate, and bit for
// bit the same x.  FCG iteration (us): 256^3 756 -> 725, 160^3 323 -> 316,
// 2048^2 241 -> 234, 1024^2 121 -> 119; below, the vectors stay in L2 and
// the pass is as long as its latency.
constexpr int64_t kDeferCells = 1 << 20;

// x += alpha p; r -= alpha q; r32 = float(r); convergence, stagnation and
// the iteration cap decide whether the loop continues.
__global__ void k_fcg_update(int64_t n, FcgState* S, bool defer, double* __restrict__ r,
                             float* __restrict__ r32, const double* P0, const double* P1,
                             const double* __restrict__ q, double* partials, double* hist,
                             int64_t hcap, Loop h) {
  pdl_enter();
  if (S->done) return;
  const long long it = S->it;
  const double alpha = S->alpha, prev = S->alpha_prev;
  double* x = S->x;
  const double* p = (it & 1) ? P1 : P0;
  double acc[1];
  if (!defer) acc[0] = fcg_update_cells<1>(n, alpha, 0.0, x, r, r32, p, nullptr, q);
  else if (it & 1) acc[0] = fcg_update_cells<2>(n, alpha, prev, x, r, r32, P1, P0, q);
  else acc[0] = fcg_update_cells<0>(n, alpha, 0.0, x, r, r32, p, nullptr, q);
  reduce_last<1>(acc, partials, &S->ticket, [&](const double* tot) {
    const double res = sqrt(tot[0]);
    const long long k = it + 1;
    S->it = k;
    S->alpha_prev = alpha;
    S->res = res;
    if (k < hcap) hist[k] = res;
    if (!isfinite(res)) {
      stop_loop(S, h, CFDB_SOLVER_NONFINITE_RESIDUAL);
      return;
    }
    if (res <= S->abs_tol || (S->b0 > 0.0 && res / S->b0 <= S->rel_tol)) {
      stop_loop(S, h, CFDB_SOLVER_CONVERGED);
      return;
    }
    if (res < S->best) {
      S->best = res;
      S->best_it = k;
    } else if (k - S->best_it >= S->window) {
      stop_loop(S, h, kLearnedStagnated);
      return;
    }
    if (k >= S->max_it) stop_loop(S, h, CFDB_SOLVER_MAX_ITERATIONS);
  });
}

// After the loop: the x update that still waits, when the last iteration
// that updated r was an even one (its direction is P0).
__global__ void k_fcg_last_x(int64_t n, const FcgState* S, const double* __restrict__ P0) {
  if (!(S->it & 1)) return;
  const double alpha = S->alpha_prev;
  double* __restrict__ x = S->x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < n; c += stride)
    x[c] = fma(alpha, P0[c], x[c]);
}

}  // namespace

// ------------------------------------------------------------------ host API

cfdb_status mg_build(cfdb_context* ctx, MgHierarchy& H, const FineOperator& op) {
  H.dim = op.dim;
  int n[3] = {op.n[0], op.n[1], op.n[2]};
  int l = 0;
  auto alloc = [&](float** p, int64_t count) -> cfdb_status {
    CFDB_CUDA(ctx, cudaMalloc((void**)p, sizeof(float) * (size_t)std::max<int64_t>(count, 4)));
    H.owned.push_back(*p);
    return CFDB_OK;
  };
  while (true) {
    MgLevel& M = H.L[l];
    std::memset(&M, 0, sizeof(M));
    for (int a = 0; a < 3; ++a) M.n[a] = n[a];
    M.cells = (int64_t)n[0] * n[1] * n[2];
    for (int a = 0; a < 3; ++a) {
      if (!axis_active(op.dim, a)) continue;
      int e[3] = {n[0], n[1], n[2]};
      e[a] += 1;
      cfdb_status rc = alloc(&M.f[a], (int64_t)e[0] * e[1] * e[2]);
      if (rc != CFDB_OK) return rc;
    }
    cfdb_status rc;
    if ((rc = alloc(&M.isq, M.cells)) != CFDB_OK || (rc = alloc(&M.res, M.cells)) != CFDB_OK)
      return rc;
    if (l > 0 && ((rc = alloc(&M.x, M.cells)) != CFDB_OK || (rc = alloc(&M.r, M.cells)) != CFDB_OK))
      return rc;
    ++l;
    int mn = 1 << 30;
    for (int a = 0; a < 3; ++a)
      if (axis_active(op.dim, a)) mn = std::min(mn, n[a]);
    const bool stop = (l > 1 && (mn <= 4 || M.cells <= 64)) || mn == 1 || l == kMgMaxLevels;
    if (stop) break;
    for (int a = 0; a < 3; ++a)
      if (axis_active(op.dim, a)) n[a] = (n[a] + 1) / 2;
  }
  H.levels = l;
  if (H.levels < 2)
    return set_error(ctx, CFDB_ERR_UNSUPPORTED, "learned preconditioner: grid too small to coarsen");
  // the block-resident tail: the longest run of levels >= 1 ending at the
  // coarsest whose levels hold at most kCoarseCells cells and whose data fit
  // in shared memory together
  int cf = H.levels - 1;
  if (coarse_bytes(H, cf) > kCoarseSmemCap)
    return set_error(ctx, CFDB_ERR_UNSUPPORTED,
                     "learned preconditioner: the coarsest level does not fit a thread block "
                     "(grid too anisotropic)");
  while (cf - 1 >= 1 && H.L[cf - 1].cells <= kCoarseCells && H.levels - (cf - 1) <= kMaxCoarse &&
         coarse_bytes(H, cf - 1) <= kCoarseSmemCap)
    --cf;
  H.coarse_from = cf;
  H.coarse_smem = coarse_bytes(H, cf);
  // opted in to the largest tail any hierarchy may have, so that hierarchies
  // of other sizes (other operators, other host threads) never lower it
  // under a launch of this one
  if (op.dim == 2)
    CFDB_CUDA(ctx, cudaFuncSetAttribute(k_coarse<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)(kCoarseSmemCap + sizeof(float) * plan_words<CoarsePlan>())));
  else
    CFDB_CUDA(ctx, cudaFuncSetAttribute(k_coarse<3>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)(kCoarseSmemCap + sizeof(float) * plan_words<CoarsePlan>())));
  return refresh_values(ctx, H, op);
}

cfdb_status mg_apply(cfdb_context* ctx, const MgHierarchy& H, const MgWeights& W, const float* r,
                     float* z, int64_t skip) {
  const int n = H.dim == 2 ? enqueue_cycle<2>(H, W, r, z, skip, nullptr, ctx->stream)
                           : enqueue_cycle<3>(H, W, r, z, skip, nullptr, ctx->stream);
  CFDB_CHECK_LAUNCH(ctx);
  count_launch(ctx, n);
  return CFDB_OK;
}

struct LearnedSolver {
  MgHierarchy* H = nullptr;
  int dim = 0;
  int n[3] = {0, 0, 0};
  int64_t cells = 0;
  uint64_t version = 0;
  MgWeights W{};
  bool have_w = false;
  double *r = nullptr, *p0 = nullptr, *p1 = nullptr, *q = nullptr, *partials = nullptr;
  float *r32 = nullptr, *z32 = nullptr;
  FcgState* S = nullptr;
  FcgState* S_host = nullptr;
  double* hist = nullptr;
  int64_t hist_cap = 0;
  cudaStream_t cap = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  int64_t launches_init = 0, launches_body = 0;
  double bytes_init = 0, bytes_iter = 0;

  void free_graph() {
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    exec = nullptr;
    graph = nullptr;
  }
  void free_all() {
    free_graph();
    delete H;
    H = nullptr;
    for (void* p : {(void*)r, (void*)p0, (void*)p1, (void*)q, (void*)partials, (void*)r32,
                    (void*)z32, (void*)S, (void*)hist})
      cudaFree(p);
    r = p0 = p1 = q = partials = nullptr;
    r32 = z32 = nullptr;
    S = nullptr;
    hist = nullptr;
    hist_cap = 0;
    if (S_host) cudaFreeHost(S_host);
    S_host = nullptr;
    if (cap) cudaStreamDestroy(cap);
    cap = nullptr;
  }
};

LearnedSolver* learned_create() {
  warm_quad_waves();
  cluster_ok(k_tail<2>);  // opt-ins and queries, before any capture
  cluster_ok(k_tail<3>);
  return new LearnedSolver();
}

void learned_destroy(LearnedSolver* s) {
  if (!s) return;
  s->free_all();
  delete s;
}

namespace {

// Blocks of the widest reduction launch (one partial per block and value):
// 2D quad passes run up to 32 blocks of 64 threads per SM.
int64_t partial_slots(const FineOperator&) { return std::max(kMaxBlocks, 148 * 32); }

template <int DIM>
void launch_init_t(LearnedSolver* s, const FineOperator& op, Loop h, cudaStream_t st) {
  const Seg sg = make_seg<DIM>(op.A.nx, op.A.ny, op.A.nz);
  launch(k_fcg_init<DIM>, seg_grid(sg), kT, 0, st, op.A, sg, s->S, s->r, s->r32, s->partials,
         s->hist, s->hist_cap, h);
}

template <int DIM>
void launch_dir_g(LearnedSolver* s, const FineOperator& op, Loop h, cudaStream_t st) {
  const res::FaceOp<DIM> A = res::face_op<DIM>(op.A, (const double*)nullptr);
  launch(k_fcg_dir_g<DIM>, gather_blocks(s->cells), 256, 0, st, A, (uint32_t)s->cells, s->S, s->z32, s->p0,
         s->p1, s->q, s->r, s->partials, h);
}

void launch_init(LearnedSolver* s, const FineOperator& op, Loop h, cudaStream_t st) {
  if (op.dim == 2) launch_init_t<2>(s, op, h, st);
  else launch_init_t<3>(s, op, h, st);
}

void launch_dir_q(LearnedSolver* s, const FineOperator& op, Loop h, cudaStream_t st) {
  const Seg sg = make_quad_seg<2>(op.A.nx, op.A.ny, op.A.nz);
  const bool tables = !op.A.fx && !op.A.fy && !op.A.fz;
  const int grid = quad_grid<2>(sg, (int64_t)dir_blocks_per_sm(tables) * 148);
  if (tables)
    launch(k_fcg_dir_q<2, true>, grid, Quad<2>::TX, 0, st, op.A, sg, s->S, s->z32, s->p0, s->p1, s->q,
           s->r, s->partials, h);
  else
    launch(k_fcg_dir_q<2, false>, grid, Quad<2>::TX, 0, st, op.A, sg, s->S, s->z32, s->p0, s->p1, s->q,
           s->r, s->partials, h);
}

void launch_dir_s(LearnedSolver* s, const FineOperator& op, Loop h, cudaStream_t st) {
  const Seg sg = make_quad_seg<3>(op.A.nx, op.A.ny, op.A.nz);
  constexpr size_t SM = dir_s_smem();
  // per-face arrays on all three axes, or the per-axis tables of a uniform operator
  if (op.A.fx && op.A.fy && op.A.fz)
    launch(k_dir_s<true>, quad_wave<3>((const void*)k_dir_s<true>, sg, SM), PlaneTile::T, SM, st,
           op.A, sg, s->S, s->z32, s->p0, s->p1, s->q, s->r, s->partials, h);
  else if (!op.A.fx && !op.A.fy && !op.A.fz)
    launch(k_dir_s<false>, quad_wave<3>((const void*)k_dir_s<false>, sg, SM), PlaneTile::T, SM, st,
           op.A, sg, s->S, s->z32, s->p0, s->p1, s->q, s->r, s->partials, h);
  else
    launch_dir_g<3>(s, op, h, st);
}

void launch_dir(LearnedSolver* s, const FineOperator& op, Loop h, cudaStream_t st) {
  if (op.dim == 2) {
    if (quad_ok<2>(op.A.nx) && s->cells > kGatherDirCells) launch_dir_q(s, op, h, st);
    else launch_dir_g<2>(s, op, h, st);
  } else {
    // 3D: the staged pass
    if (quad_ok<3>(op.A.nx)) launch_dir_s(s, op, h, st);
    else launch_dir_g<3>(s, op, h, st);
  }
}

bool defers(const LearnedSolver* s) { return s->cells >= kDeferCells; }

// One FCG iteration: V-cycle z = M r (its last kernel also forms z.q and
// beta), direction + A p, update.  Returns the number of kernels.
int enqueue_body(LearnedSolver* s, const FineOperator& op, Loop h, cudaStream_t st) {
  const int64_t skip = op.pinned ? op.ref : -1;
  const Hook hk{s->q, s->partials, s->S, h};
  const int nv = op.dim == 2 ? enqueue_cycle<2>(*s->H, s->W, s->r32, s->z32, skip, &hk, st)
                             : enqueue_cycle<3>(*s->H, s->W, s->r32, s->z32, skip, &hk, st);
  launch_dir(s, op, h, st);
  launch(k_fcg_update, flat_grid(s->cells), 256, 0, st, s->cells, s->S, defers(s), s->r, s->r32, s->p0,
         s->p1, s->q, s->partials, s->hist, s->hist_cap, h);
  return nv + 2;
}

// Solve loop without a graph, for profilers that cannot look inside graphs
// with conditional nodes (CFDB_LEARNED_LAUNCH=stream): the same kernels,
// launched per iteration, the host reading the state after each iteration.
cfdb_status run_stream_mode(cfdb_context* ctx, LearnedSolver* s, const FineOperator& op) {
  launch_init(s, op, Loop{0, 0}, ctx->stream);
  CFDB_CHECK_LAUNCH(ctx);
  while (true) {
    CFDB_CUDA(ctx, cudaMemcpyAsync(s->S_host, s->S, sizeof(FcgState), cudaMemcpyDeviceToHost,
                                   ctx->stream));
    CFDB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (s->S_host->done) break;
    enqueue_body(s, op, Loop{0, 0}, ctx->stream);
    CFDB_CHECK_LAUNCH(ctx);
  }
  return CFDB_OK;
}

void count_bytes(LearnedSolver* s, const FineOperator& op) {
  // algorithmic bytes: the start (b, x in; r, r32 out) and per iteration the
  // V-cycle, the direction pass (z, p_old, r in; p, q out), the update (x, p,
  // r, q in; x, r, r32 out; a deferred x half as often, with two p) and the
  // z.q read of q; face arrays when present
  int face_words = 0;
  for (int a = 0; a < 3; ++a) face_words += op.full[a] ? 1 : 0;
  const double n = (double)s->cells;
  s->bytes_init = n * (8.0 * (3 + face_words) + 4.0);
  s->bytes_iter = cycle_bytes(*s->H, s->W) + n * (4.0 + 8.0 * (4 + face_words)) +
                  n * (8.0 * (defers(s) ? 5 : 6) + 4.0) + n * 8.0;
}

// The layout of a system's FCG in one cluster (words = 0: too large, no such
// cluster, or the profilers' launch-by-launch mode).
ClusterLayout fcg_layout(const LearnedSolver* s) {
  const char* mode = std::getenv("CFDB_LEARNED_LAUNCH");
  if (s->cells > kFcgClusterCells || (mode && std::strcmp(mode, "stream") == 0) ||
      !(s->dim == 2 ? cluster_ok(k_fcg_cluster<2>) : cluster_ok(k_fcg_cluster<3>)))
    return ClusterLayout{};
  return cluster_layout(*s->H, s->W, 0, true, nullptr, nullptr);
}

cfdb_status run_in_cluster(cfdb_context* ctx, LearnedSolver* s, const FineOperator& op,
                           const ClusterLayout& C) {
  FcgArgs F;
  std::memset(&F, 0, sizeof(F));
  F.A = op.A;
  F.S = s->S;
  F.hist = s->hist;
  F.hcap = s->hist_cap;
  F.pin = op.pinned ? (int)op.ref : -1;
  const size_t smem = sizeof(float) * (size_t)C.words;
  const cudaError_t e =
      s->dim == 2 ? res::launch_cluster(k_fcg_cluster<2>, res::kMaxCluster, res::kMaxCluster, kClusterT,
                                        smem, ctx->stream, F, C.P, C.Q, C.words)
                  : res::launch_cluster(k_fcg_cluster<3>, res::kMaxCluster, res::kMaxCluster, kClusterT,
                                        smem, ctx->stream, F, C.P, C.Q, C.words);
  if (e != cudaSuccess) return cuda_error(ctx, e, "learned solve in a cluster", __FILE__, __LINE__);
  return CFDB_OK;
}

cfdb_status capture_graph(cfdb_context* ctx, LearnedSolver* s, const FineOperator& op) {
  s->free_graph();
  CFDB_CUDA(ctx, cudaGraphCreate(&s->graph, 0));
  cudaGraphConditionalHandle h;
  CFDB_CUDA(ctx, cudaGraphConditionalHandleCreate(&h, s->graph, 1, cudaGraphCondAssignDefault));
  // parent graph: the initial residual, then the WHILE node
  take_launch_error();
  CFDB_CUDA(ctx, cudaStreamBeginCaptureToGraph(s->cap, s->graph, nullptr, nullptr, 0,
                                               cudaStreamCaptureModeThreadLocal));
  const Loop lp{h, 1};
  launch_init(s, op, lp, s->cap);
  cudaGraph_t g = nullptr;
  cudaError_t ce = cudaStreamEndCapture(s->cap, &g);
  if (ce == cudaSuccess) ce = take_launch_error();
  if (ce != cudaSuccess) return cuda_error(ctx, ce, "capture of the FCG start", __FILE__, __LINE__);
  size_t nn = 0;
  CFDB_CUDA(ctx, cudaGraphGetNodes(s->graph, nullptr, &nn));
  if (nn != 1) return set_error(ctx, CFDB_ERR_CUDA, "unexpected FCG start graph");
  cudaGraphNode_t init_node;
  CFDB_CUDA(ctx, cudaGraphGetNodes(s->graph, &init_node, &nn));
  cudaGraphNodeParams cp = {cudaGraphNodeTypeConditional};
  cp.conditional.handle = h;
  cp.conditional.type = cudaGraphCondTypeWhile;
  cp.conditional.size = 1;
  cudaGraphNode_t loop_node;
  CFDB_CUDA(ctx, cudaGraphAddNode(&loop_node, s->graph, &init_node, 1, &cp));
  cudaGraph_t body = cp.conditional.phGraph_out[0];
  // body: one FCG iteration
  CFDB_CUDA(ctx, cudaStreamBeginCaptureToGraph(s->cap, body, nullptr, nullptr, 0,
                                               cudaStreamCaptureModeThreadLocal));
  const int nv = enqueue_body(s, op, lp, s->cap);
  cudaGraph_t b2 = nullptr;
  ce = cudaStreamEndCapture(s->cap, &b2);
  if (ce == cudaSuccess) ce = take_launch_error();
  if (ce != cudaSuccess) return cuda_error(ctx, ce, "capture of the FCG loop", __FILE__, __LINE__);
  CFDB_CHECK_LAUNCH(ctx);
  CFDB_CUDA(ctx, cudaGraphInstantiate(&s->exec, s->graph, 0));
  s->launches_init = 1;
  s->launches_body = nv;
  return CFDB_OK;
}

}  // namespace

namespace {

// Builds (new shape) or refreshes (new coefficient version) the hierarchy and
// the FCG vectors; *recapture tells whether the solve graph must be rebuilt.
cfdb_status ensure_state(cfdb_context* ctx, LearnedSolver* s, const FineOperator& op,
                         uint64_t version, bool* recapture_out) {
  const int64_t cells = (int64_t)op.n[0] * op.n[1] * op.n[2];
  const bool same_shape = s->H && s->dim == op.dim && s->n[0] == op.n[0] && s->n[1] == op.n[1] &&
                          s->n[2] == op.n[2];
  bool recapture = false;
  if (!same_shape) {
    s->free_all();
    s->H = new MgHierarchy();
    s->dim = op.dim;
    for (int a = 0; a < 3; ++a) s->n[a] = op.n[a];
    s->cells = cells;
    cfdb_status st = mg_build(ctx, *s->H, op);
    auto a64 = [&](double** p, int64_t m) -> cfdb_status {
      CFDB_CUDA(ctx, cudaMalloc((void**)p, sizeof(double) * (size_t)m));
      return CFDB_OK;
    };
    auto a32 = [&](float** p, int64_t m) -> cfdb_status {
      CFDB_CUDA(ctx, cudaMalloc((void**)p, sizeof(float) * (size_t)m));
      return CFDB_OK;
    };
    if (st != CFDB_OK || (st = a64(&s->r, cells)) != CFDB_OK || (st = a64(&s->p0, cells)) != CFDB_OK ||
        (st = a64(&s->p1, cells)) != CFDB_OK || (st = a64(&s->q, cells)) != CFDB_OK ||
        (st = a64(&s->partials, 2 * partial_slots(op))) != CFDB_OK ||
        (st = a32(&s->r32, cells)) != CFDB_OK || (st = a32(&s->z32, cells)) != CFDB_OK) {
      s->free_all();
      return st;
    }
    // cleared on the context's own stream: the context streams are
    // non-blocking, so a legacy-stream memset would not be ordered before the
    // solve's own writes of the state (and could land after them)
    cudaError_t e1 = cudaMalloc((void**)&s->S, sizeof(FcgState));
    cudaError_t e2 =
        e1 == cudaSuccess ? cudaMemsetAsync(s->S, 0, sizeof(FcgState), ctx->stream) : e1;
    cudaError_t e3 =
        e2 == cudaSuccess ? cudaMemsetAsync(s->q, 0, sizeof(double) * cells, ctx->stream) : e2;
    cudaError_t e4 = e3 == cudaSuccess ? cudaMallocHost((void**)&s->S_host, sizeof(FcgState)) : e3;
    cudaError_t e5 = e4 == cudaSuccess ? cudaStreamCreateWithFlags(&s->cap, cudaStreamNonBlocking) : e4;
    if (e5 != cudaSuccess) {
      s->free_all();
      return cuda_error(ctx, e5, "learned solver state", __FILE__, __LINE__);
    }
    s->version = version;
    recapture = true;
  } else if (s->version != version) {
    cfdb_status st = refresh_values(ctx, *s->H, op);
    if (st != CFDB_OK) return st;
    s->version = version;
  }
  *recapture_out = recapture;
  return CFDB_OK;
}

}  // namespace

cfdb_status learned_hierarchy(cfdb_context* ctx, LearnedSolver* s, const FineOperator& op,
                              uint64_t version, const MgHierarchy** out) {
  bool recapture = false;
  cfdb_status st = ensure_state(ctx, s, op, version, &recapture);
  if (st != CFDB_OK) return st;
  if (recapture) s->free_graph();
  *out = s->H;
  return CFDB_OK;
}

cfdb_status learned_solve(cfdb_context* ctx, LearnedSolver* s, const FineOperator& op,
                          uint64_t version, const MgWeights& W, const double* b, double* x,
                          double abs_tol, double rel_tol, int64_t max_it, int64_t hist_cap,
                          LearnedOutcome* out) {
  std::memset(out, 0, sizeof(*out));
  bool recapture = false;
  {
    cfdb_status st = ensure_state(ctx, s, op, version, &recapture);
    if (st != CFDB_OK) return st;
  }
  const int64_t want_hist = std::max<int64_t>(hist_cap, 1);
  if (s->hist_cap < want_hist) {
    cudaFree(s->hist);
    s->hist = nullptr;
    s->hist_cap = 0;
    CFDB_CUDA(ctx, cudaMalloc((void**)&s->hist, sizeof(double) * (size_t)want_hist));
    s->hist_cap = want_hist;
    recapture = true;
  }
  if (!s->have_w || std::memcmp(&s->W, &W, sizeof(W)) != 0) {
    s->W = W;
    s->have_w = true;
    recapture = true;
  }
  const ClusterLayout CL = fcg_layout(s);
  const bool in_cluster = CL.words > 0;
  if (recapture) s->free_graph();
  if (!in_cluster && !s->exec) {
    cfdb_status st = capture_graph(ctx, s, op);
    if (st != CFDB_OK) {
      s->free_graph();
      return st;
    }
  }
  count_bytes(s, op);
  FcgState& hs = *s->S_host;
  std::memset(&hs, 0, sizeof(hs));
  hs.b = b;
  hs.x = x;
  hs.abs_tol = abs_tol;
  hs.rel_tol = rel_tol;
  hs.max_it = max_it;
  hs.window = 50;
  hs.status = kRunning;
  CFDB_CUDA(ctx, cudaMemcpyAsync(s->S, &hs, sizeof(FcgState), cudaMemcpyHostToDevice, ctx->stream));
  CFDB_CUDA(ctx, cudaEventRecord(ctx->ev_k0, ctx->stream));
  const char* mode = std::getenv("CFDB_LEARNED_LAUNCH");
  if (in_cluster) {
    cfdb_status st = run_in_cluster(ctx, s, op, CL);
    if (st != CFDB_OK) return st;
  } else if (mode && std::strcmp(mode, "stream") == 0) {
    cfdb_status st = run_stream_mode(ctx, s, op);
    if (st != CFDB_OK) return st;
  } else {
    CFDB_CUDA(ctx, cudaGraphLaunch(s->exec, ctx->stream));
  }
  const bool last_x = !in_cluster && defers(s);
  if (last_x) {
    k_fcg_last_x<<<flat_grid(s->cells), 256, 0, ctx->stream>>>(s->cells, s->S, s->p0);
    CFDB_CHECK_LAUNCH(ctx);
  }
  CFDB_CUDA(ctx, cudaEventRecord(ctx->ev_k1, ctx->stream));
  CFDB_CUDA(ctx, cudaMemcpyAsync(s->S_host, s->S, sizeof(FcgState), cudaMemcpyDeviceToHost, ctx->stream));
  CFDB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  float ms = 0.f;
  CFDB_CUDA(ctx, cudaEventElapsedTime(&ms, ctx->ev_k0, ctx->ev_k1));
  out->status = hs.status;
  out->iterations = hs.it;
  out->initial_residual = hs.b0;
  out->final_residual = hs.res;
  out->kernel_ms = ms;
  out->bytes = s->bytes_init + s->bytes_iter * (double)hs.it;
  if (last_x && (hs.it & 1)) out->bytes += 8.0 * (double)s->cells;
  out->launches =
      in_cluster ? 1 : s->launches_init + s->launches_body * hs.it + (last_x ? 1 : 0);
  count_launch(ctx, (int)std::min<int64_t>(out->launches, 1 << 30));
  return CFDB_OK;
}

cfdb_status learned_history(cfdb_context* ctx, LearnedSolver* s, double* host, int64_t m) {
  if (!s->hist || m <= 0) return CFDB_OK;
  m = std::min(m, s->hist_cap);
  CFDB_CUDA(ctx, cudaMemcpyAsync(host, s->hist, sizeof(double) * (size_t)m, cudaMemcpyDeviceToHost,
                                 ctx->stream));
  CFDB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return CFDB_OK;
}

namespace {
struct CtxWeights {
  MgWeights w[2];
};
void free_ctx_weights(void* p) { delete static_cast<CtxWeights*>(p); }

CtxWeights& ctx_weights(cfdb_context* ctx) {
  if (!ctx->mg_weights) {
    auto* cw = new CtxWeights();
    cw->w[0] = mg_builtin_weights(2);
    cw->w[1] = mg_builtin_weights(3);
    ctx->mg_weights = cw;
    ctx->mg_weights_free = free_ctx_weights;
  }
  return *static_cast<CtxWeights*>(ctx->mg_weights);
}
}  // namespace

const MgWeights& mg_context_weights(cfdb_context* ctx, int dim) {
  return ctx_weights(ctx).w[dim == 3 ? 1 : 0];
}

}  // namespace cfdb

using namespace cfdb;

extern "C" {

cfdb_status cfdb_mg_set_weights(cfdb_context* ctx, int dim, int levels, int nu, int coarse_sweeps,
                                const float* kernels, const float* coarse_weights) {
  if (!ctx || !kernels || !coarse_weights) return CFDB_ERR_INVALID_ARGUMENT;
  if (levels < 1 || levels > kMgMaxLevels)
    return set_error(ctx, CFDB_ERR_INVALID_ARGUMENT, "weights: levels must be 1..16");
  MgWeights W = mg_default_weights(dim);
  W.levels = levels;
  W.nu = nu;
  W.coarse_sweeps = coarse_sweeps;
  for (int l = 0; l < kMgMaxLevels; ++l) {
    const int src = std::min(l, levels - 1);
    for (int t = 0; t < kMgTaps; ++t) W.w[l][t] = kernels[src * kMgTaps + t];
    W.c[l] = coarse_weights[src];
  }
  std::string why;
  if (!mg_weights_valid(W, &why)) return set_error(ctx, CFDB_ERR_INVALID_ARGUMENT, why);
  ctx_weights(ctx).w[dim == 3 ? 1 : 0] = W;
  return CFDB_OK;
}

cfdb_status cfdb_mg_get_weights(cfdb_context* ctx, int dim, int* levels, int* nu,
                                int* coarse_sweeps, float* kernels, float* coarse_weights) {
  if (!ctx || (dim != 2 && dim != 3)) return CFDB_ERR_INVALID_ARGUMENT;
  const MgWeights& W = mg_context_weights(ctx, dim);
  if (levels) *levels = W.levels;
  if (nu) *nu = W.nu;
  if (coarse_sweeps) *coarse_sweeps = W.coarse_sweeps;
  if (kernels) std::memcpy(kernels, W.w, sizeof(W.w));
  if (coarse_weights) std::memcpy(coarse_weights, W.c, sizeof(W.c));
  return CFDB_OK;
}

cfdb_status cfdb_mg_apply(cfdb_context* ctx, cfdb_poperator* op, const float* r_host,
                          float* z_host) {
  if (!ctx || !op || !r_host || !z_host) return CFDB_ERR_INVALID_ARGUMENT;
  CFDB_CUDA(ctx, cudaSetDevice(ctx->device));
  FineOperator fo;
  LearnedSolver* solver = nullptr;
  uint64_t version = 0;
  poperator_learned(op, &fo, &solver, &version);
  const MgHierarchy* H = nullptr;
  cfdb_status st = learned_hierarchy(ctx, solver, fo, version, &H);
  if (st != CFDB_OK) return st;
  const int64_t n = H->L[0].cells;
  float *r = nullptr, *z = nullptr;
  CFDB_CUDA(ctx, cudaMalloc((void**)&r, sizeof(float) * n));
  if (cudaMalloc((void**)&z, sizeof(float) * n) != cudaSuccess) {
    cudaFree(r);
    return set_error(ctx, CFDB_ERR_OUT_OF_MEMORY, "mg_apply buffers");
  }
  cudaStream_t s = ctx->stream;
  cudaError_t e = cudaMemcpyAsync(r, r_host, sizeof(float) * n, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) {
    st = mg_apply(ctx, *H, mg_context_weights(ctx, fo.dim), r, z, fo.pinned ? fo.ref : -1);
    if (st == CFDB_OK) e = cudaMemcpyAsync(z_host, z, sizeof(float) * n, cudaMemcpyDeviceToHost, s);
    if (st == CFDB_OK && e == cudaSuccess) e = cudaStreamSynchronize(s);
  }
  cudaFree(r);
  cudaFree(z);
  if (e != cudaSuccess) return cuda_error(ctx, e, "mg_apply", __FILE__, __LINE__);
  return st;
}

cfdb_status cfdb_mg_reset_weights(cfdb_context* ctx, int dim, int trained) {
  if (!ctx || (dim != 2 && dim != 3)) return CFDB_ERR_INVALID_ARGUMENT;
  ctx_weights(ctx).w[dim == 3 ? 1 : 0] = trained ? mg_builtin_weights(dim) : mg_default_weights(dim);
  return CFDB_OK;
}

}  // extern "C"
