"""Device routines that a host compiler takes (device_on_host.h), run on the CPU
with a team of one block and one thread that records what the team is asked to do.
"""
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
