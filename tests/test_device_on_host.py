"""Device routines that a host compiler takes (device_on_host.h), run on the CPU
with a team of one block and one thread that records what the team is asked to do.
"""
import math
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "cfdapp_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def _run(tmp_path, source):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(source)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-w", "-ffp-contract=off", "-I", HERE,
                           "-I", CSRC, "-I", os.path.join(ROOT, "include"),
                           "-I", os.path.join(CUDA, "include"), str(src), "-o", str(exe)])
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True,
                          timeout=120).stdout.split()


# a 4 x 3 system, diagonally dominant and not symmetric
KRYLOV = r"""
#include "device_on_host.h"
#include "resident.cuh"
#include <cstdio>
#include <string>
using namespace cfdb;
struct Team {
  static constexpr bool kGlobal = false;
  std::string ops;
  int rank() const { return 0; }
  void enter() { ops += 'e'; }
  bool sync() { ops += 's'; return true; }
  template <int NV> bool reduce(double (&v)[NV]) { ops += (char)('0' + NV); return true; }
  double remote(const double* v, const double*, uint32_t c) const { return v[c]; }
};
int main() {
  const int nx = 4, ny = 3, n = 12;
  double diag[12], off[4][12], b[12], x[12], out[8], sm[12 * 8];
  for (int c = 0; c < n; ++c) {
    diag[c] = 4.0 + 0.01 * c;
    for (int q = 0; q < 4; ++q) off[q][c] = -1.0 + (SYM ? 0.0 : 0.05 * q);
    b[c] = sin(1.0 + c);
    x[c] = 0.0;
  }
  StencilMatrix M{};
  M.dim = 2; M.nx = nx; M.ny = ny; M.nz = 1; M.n = n; M.sy = nx; M.sz = n;
  M.diag = diag;
  for (int q = 0; q < 4; ++q) M.off[q] = off[q];
  res::Io P{};
  P.b = b; P.x = x; P.rel_tol = 1e-12; P.max_it = 50; P.out = out;
  Team T;
  RUN
  printf("%s %d\n", T.ops.c_str(), (int)out[0]);
}
"""


@pytest.mark.parametrize("sym,run", [
    (1, "res::cg_run<1, 12, true, true, true>(res::band_op<2>(M), (uint32_t)n, (uint32_t)n, P, T, sm);"),
    (1, "res::cg_run<1, 12, false, true, true>(res::band_op<2>(M), (uint32_t)n, (uint32_t)n, P, T, sm);"),
    (0, "res::bicgstab_run<1, 0, true, false>(res::band_op<2>(M), (uint32_t)n, (uint32_t)n, P, T, sm);"),
])
def test_cluster_solves_enter_the_team_first(tmp_path, sym, run):
    """A cluster's block may store into another's shared memory (a reduction does) only once
    that block has started: the first thing asked of the team is that every block enters."""
    ops, status = _run(tmp_path, KRYLOV.replace("RUN", run).replace("SYM", str(sym)))
    assert status == "0"  # converged
    assert ops[0] == "e", ops


# measured solve stages of one outer iteration on the GPU (ms, clusters and teams): dimension,
# side, cases, method, p' system or momentum
STAGES = [(2, 48, 7, 0, 1, 0.98, 4.7), (2, 48, 64, 0, 1, 9.7, 4.9), (2, 96, 24, 0, 1, 8.9, 13.8),
          (2, 96, 64, 0, 1, 22.2, 14.5), (2, 128, 16, 0, 1, 9.4, 17.7), (2, 128, 32, 0, 1, 15.6, 18.6),
          (2, 128, 64, 0, 1, 31.1, 22.9), (2, 192, 16, 0, 1, 23.9, 27.0),
          (2, 256, 16, 0, 1, 40.4, 46.7), (2, 256, 32, 0, 1, 67.5, 99.4),
          (3, 16, 64, 0, 1, 5.8, 3.9), (3, 33, 16, 0, 1, 8.8, 10.9), (3, 33, 32, 0, 1, 14.6, 17.3),
          (3, 33, 48, 0, 1, 20.5, 21.9),
          (2, 128, 32, 1, 1, 39.4, 29.1), (2, 128, 16, 1, 1, 23.6, 27.7),
          (2, 48, 7, 1, 0, 0.41, 1.15), (2, 48, 32, 1, 0, 1.98, 1.18), (2, 128, 64, 1, 0, 4.09, 2.17),
          (2, 256, 16, 1, 0, 1.90, 2.21), (2, 256, 32, 1, 0, 3.18, 3.98),
          (3, 24, 32, 1, 0, 3.49, 2.24), (3, 24, 8, 1, 0, 1.40, 2.16)]


def test_batches_take_clusters_where_they_were_faster(tmp_path):
    """The choice between one cluster per case and block teams, against both sides measured."""
    rows = "".join(f"{{{d},{s},{c},{k},{p}}}," for d, s, c, k, p, _, _ in STAGES)
    got = _run(tmp_path, r"""
#include "device_on_host.h"
#include "resident_launch.cuh"
#include <cstdio>
int main() {
  const int rows[][5] = {""" + rows + r"""};
  for (auto& r : rows) {
    const int64_t n = r[0] == 2 ? (int64_t)r[1] * r[1] : (int64_t)r[1] * r[1] * r[1];
    std::vector<int64_t> side(r[2], r[1]), cells(r[2], n);
    printf("%d ", (int)cfdb::res::clusters_pay(r[0], r[2], side.data(), cells.data(), r[3], r[4]));
  }
}
""")
    for row, pay in zip(STAGES, got):
        assert (pay == "1") == (row[5] < row[6]), row


def test_bicgstab_dot_products_round_once(tmp_path):
    """The three dot products of an iteration -- (rHat, v), (t, s) and (rHat, r) -- as sums of
    fused multiply-adds: a single-thread team sees the sums and the vectors they are of."""
    team = r"""
struct Team {
  static constexpr bool kGlobal = false;
  const double *rh, *v, *r, *t;
  int n, triple = 0, bad = 0, seen = 0;
  int rank() const { return 0; }
  void enter() {}
  bool sync() { return true; }
  double dot(const double* a, const double* b) const {
    double s = 0.0;
    for (int c = 0; c < n; ++c) s = fma(a[c], b[c], s);
    return s;
  }
  template <int NV> bool reduce(double (&o)[NV]) {
    if (NV != 3) return true;
    const double want[3] = {dot(rh, v), dot(t, r), dot(rh, r)};
    ++seen;
    bad += o[triple == 0 ? 0 : 1] != want[triple];
    triple = (triple + 1) % 3;
    return true;
  }
  double remote(const double* q, const double*, uint32_t c) const { return q[c]; }
};
int main() {"""
    src = KRYLOV.replace(KRYLOV[KRYLOV.index("struct Team"):KRYLOV.index("int main() {") + 12], team)
    src = src.replace("SYM", "0").replace("RUN", r"""
  T.n = n; T.r = sm + n; T.rh = sm + 2 * n; T.v = sm + 3 * n; T.t = sm + 4 * n;
  res::bicgstab_run<1, 0, true, false>(res::band_op<2>(M), (uint32_t)n, (uint32_t)n, P, T, sm);
""").replace(r'printf("%s %d\n", T.ops.c_str(), (int)out[0]);', r'printf("%d %d\n", T.seen, T.bad);')
    seen, bad = _run(tmp_path, src)
    assert int(seen) >= 9 and bad == "0", (seen, bad)


# measured CG iterations on the GPU (us, cluster and grid): dimension, cells, plane
LINE = [(2, 22500, 150, 4.9, 5.9), (2, 32761, 181, 5.65, 5.92), (2, 33124, 182, 6.05, 5.74),
        (2, 36100, 190, 6.11, 5.76), (3, 24389, 841, 6.1, 6.4), (3, 27000, 900, 6.7, 6.4),
        (3, 35937, 1089, 7.3, 6.3)]


def test_cg_takes_the_team_that_was_faster(tmp_path):
    got = _run(tmp_path, r"""
#include "device_on_host.h"
#include "resident_launch.cuh"
#include <cstdio>
using namespace cfdb::res;
int main() {
  const int rows[][3] = {""" + "".join(f"{{{d},{n},{h}}}," for d, n, h, _, _ in LINE) + r"""};
  for (auto& r : rows)
    printf("%d ", cg_plan(r[1], r[2], 148, r[1] <= cluster_cells(r[0]) ? 16 : 0).team);
}
""")
    for row, team in zip(LINE, got):
        assert team == ("1" if row[3] < row[4] else "2"), row


@pytest.mark.parametrize("n,nx,ny", [(46339 * 46339, 46339, 1), (1290 ** 3, 1290, 1290), (1 << 31, 2, 1 << 20),
                                     (1000, 10, 10)])
def test_gathering_passes_end_at_the_last_cell(tmp_path, n, nx, ny):
    """The one-cell-per-thread loop of the largest grids, as the first and the last thread of a
    full launch run it: every index below n, the right coordinates, and no step past the end."""
    got = _run(tmp_path, r"""
#include "device_on_host.h"
#include "cell_index.cuh"
#include <cstdio>
int main() {
  const uint32_t n = %du; const int nx = %d, ny = %d;
  gridDim.x = 2368;
  for (int last = 0; last < 2; ++last) {
    blockIdx.x = last ? gridDim.x - 1 : 0;
    threadIdx.x = last ? 255 : 0;
    long long count = 0, bad = 0, top = -1;
    cfdb::res::gather_cells(n, nx, ny, cfdb::res::fast_div(nx), cfdb::res::fast_div(ny),
                            [&](uint32_t c, int i, int j, int k) {
      bad += c >= n || i < 0 || i >= nx || j < 0 || j >= ny || k < 0;
      bad += (uint32_t)(i + (long long)nx * (j + (long long)ny * k)) != c;
      top = c;
      if (++count > 10000) { printf("runaway\n"); std::exit(0); }
    });
    printf("%%lld %%lld %%lld ", count, top, bad);
  }
}
""" % (n, nx, ny))
    stride = 2368 * 256
    for first, (count, top, bad) in zip((0, stride - 1), (map(int, got[:3]), map(int, got[3:]))):
        want = max(0, -(-(n - first) // stride))
        assert (count, bad) == (want, 0)
        assert top == (first + (want - 1) * stride if want else -1)


# the plans behind the grids of test_large_gpu.py on 148 SMs: system, bytes of a word, method
# (0 CG, 1 BiCGSTAB) -> team, most cells a thread, x and the neighbouring planes on chip
PLANS = [((787, 773), 8, 0, (2, 5, 1, 1)), ((89, 83, 84), 8, 0, (2, 5, 1, 1)),
         ((1123, 1117), 8, 0, (2, 9, 1, 1)), ((109, 107, 105), 8, 0, (2, 9, 1, 0)),
         ((1231, 1229), 8, 0, (2, 10, 0, 1)), ((115, 115, 115), 8, 0, (2, 11, 0, 0)),
         ((128, 128, 128), 8, 0, (2, 14, 0, 0)), ((1460, 1456), 8, 0, None), ((1459, 1457), 8, 0, None),
         ((132, 128, 126), 8, 0, None), ((131, 129, 127), 8, 0, None),
         ((640, 500), 8, 0, (2, 3, 1, 1)), ((128, 128, 32), 8, 0, (2, 4, 1, 0)),
         ((128, 116, 104), 8, 0, (2, 11, 0, 0)), ((203, 201), 4, 0, (2, 1, 1, 1)),
         ((45, 43, 41), 4, 0, (2, 2, 1, 1)), ((703, 433), 4, 0, (2, 3, 1, 1)),
         ((181, 161, 11), 4, 0, (2, 3, 1, 0)), ((125, 121, 119), 4, 0, (2, 12, 0, 1)),
         ((1459, 1457), 4, 0, None), ((131, 129, 127), 4, 0, None),
         ((887, 853), 8, 1, (2, 10, 0, 0)), ((93, 91, 89), 8, 1, (2, 10, 0, 0)),
         ((951, 901), 8, 1, None), ((97, 95, 93), 8, 1, None)]


def test_plans_of_large_systems(tmp_path):
    rows = "".join("{%d,%d,%d,%d}," % (int(math.prod(n)), n[0] if len(n) == 2 else n[0] * n[1],
                                       word, krylov) for n, word, krylov, _ in PLANS)
    got = _run(tmp_path, r"""
#include "device_on_host.h"
#include "resident_launch.cuh"
#include <cstdio>
using namespace cfdb::res;
int main() {
  const int rows[][4] = {""" + rows + r"""};
  for (auto& r : rows) {
    const Plan P = r[3] == 1 ? bicgstab_plan(r[0], 148, 0) : cg_plan(r[0], r[1], 148, 0, r[2]);
    printf("%d %d %d %d ", P.team, P.nc, (int)P.xs, (int)P.halo);
  }
}
""")
    got = [tuple(map(int, got[4 * q:4 * q + 4])) for q in range(len(PLANS))]
    for row, g in zip(PLANS, got):
        if row[3] is None:
            assert g[0] == 0, (row, g)
        else:
            assert g == row[3], (row, g)
