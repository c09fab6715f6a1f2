"""The solves of large systems against the CPU oracle: the on-chip kernels' larger variants (eight
and fourteen cells a thread, x in memory, no neighbouring planes) and, past what the chip holds,
the streaming kernels -- tiled by TMA and plain, tables and face arrays, FP64 and FP32.

FP64 iterates after a fixed number of iterations agree to rounding (1e-10 relative L2, histories
1e-8, as in test_resident_gpu.py).  The FP32-refined forms run the same iterations with FP32
directions: each rounds p, z (and r) once, 6e-8 relative, so that six iterations of some ten
roundings each stay within 2e-5 of the update.
"""
import numpy as np
import pytest

from oracle import oracle as O
from test_resident_gpu import _csr, _rel, _system

pytestmark = pytest.mark.gpu

# on chip: variants that smaller grids do not reach
CHIP = [(787, 773), (89, 83, 84), (1123, 1117), (109, 107, 105), (1231, 1229), (115, 115, 115),
        (128, 128, 128)]
# past the chip: rows that the TMA kernel takes, and rows that it does not
STREAM = [(1460, 1456), (1459, 1457), (132, 128, 126), (131, 129, 127)]


def _run(ctx, n, precision, uniform=False, its=6):
    from cfdapp_b200.cfdb import LinearSolverSettings, POperator
    dim, length = len(n), tuple(float(m) for m in n)
    rng = np.random.default_rng(12)
    if uniform:
        case = O.Case(dim, n, length, [("wall", (0, 0, 0))] * (2 * dim),
                      [("fixed_gradient", 0.0)] * (2 * dim))
        ones = np.ones(case.cells())
        _, diag, off, _ = O.assemble_pprime(case, 1.0, np.zeros(case.faces()), ones, ones, ones)
        rhs = rng.normal(size=case.cells())
        op = POperator(ctx, dim, n, length)
    else:
        case, fc, diag, off, rhs = _system(n, 11, True)
        op = POperator(ctx, dim, n, length, face_coeff=fc, pinned=False)
    x0 = rng.normal(size=case.cells())
    ref = O.stencil_solve(case, diag, off, rhs, x0=x0, rel_tol=1e-30, max_iterations=its)
    got = op.solve(rhs, LinearSolverSettings(absolute_tolerance=0.0, relative_tolerance=1e-30,
                                             max_iterations=its, precision=precision), x0=x0)
    op.close()
    return case, diag, off, rhs, x0, ref, got


@pytest.mark.parametrize("n", CHIP + STREAM)
@pytest.mark.parametrize("uniform", [False, True])
def test_pcg_iterates_match_oracle(ctx, n, uniform):
    _, _, _, _, _, ref, got = _run(ctx, n, "fp64", uniform)
    assert got.status == ref.status and got.iterations == ref.iterations
    np.testing.assert_allclose(got.residual_history, ref.history, rtol=1e-8)
    assert _rel(got.solution, ref.solution) <= 1e-10


# mixed precision (rows of a multiple of four): 1024-thread blocks, no neighbouring planes, x in
# memory, and the streaming kernel; FP32 refinement (other rows): both block sizes of the grid
# team, no neighbouring planes, x in memory, and the streaming kernel
@pytest.mark.parametrize("n", [(640, 500), (128, 128, 32), (128, 116, 104), (1460, 1456), (132, 128, 126),
                               (203, 201), (45, 43, 41), (703, 433), (181, 161, 11), (125, 121, 119),
                               (1459, 1457), (131, 129, 127)])
@pytest.mark.parametrize("uniform", [False, True])
def test_fp32_refined_iterates_follow_the_fp64_ones(ctx, n, uniform):
    case, diag, off, rhs, x0, ref, got = _run(ctx, n, "fp32_refined", uniform)
    assert got.iterations == ref.iterations and got.refinements >= 1
    assert np.linalg.norm(got.solution - ref.solution) <= 2e-5 * np.linalg.norm(ref.solution - x0)
    true = np.linalg.norm(rhs - O.stencil_apply(case, diag, off, got.solution))
    assert got.true_residual == pytest.approx(true, rel=1e-9)


# BiCGSTAB on chip with x in memory and streaming, CG on chip with x in memory and streaming
@pytest.mark.parametrize("n,method", [((887, 853), "bicgstab"), ((93, 91, 89), "bicgstab"),
                                      ((951, 901), "bicgstab"), ((97, 95, 93), "bicgstab"),
                                      ((1231, 1229), "cg"), ((115, 115, 115), "cg"), ((1459, 1457), "cg"),
                                      ((131, 129, 127), "cg")])
@pytest.mark.parametrize("jacobi", [False, True])
def test_band_solves_match_oracle(ctx, n, method, jacobi):
    import test_resident_gpu
    test_resident_gpu.test_band_solves_match_oracle(ctx, n, method, jacobi)


# copies of a 3-cell system whose first BiCGSTAB residual has no part along rHat (their supports
# are disjoint, so (rHat, r) is 0 whatever the order of the sum): rho vanishes, the solve restarts
# from its iterate and converges.  One block, a cluster, the grid with x on chip and in memory, and
# streaming.
@pytest.mark.parametrize("copies", [40, 9000, 100000, 250000, 300000])
def test_bicgstab_restart_matches_oracle(ctx, copies):
    from cfdapp_b200.cfdb import CsrSolver, LinearSolverSettings
    n = (3, copies)
    case = O.Case(2, n, (3.0, float(copies)), [("wall", (0, 0, 0))] * 4, [("fixed_gradient", 0.0)] * 4)
    diag, lo, hi, b = (np.tile(np.array(v), copies) for v in
                       ([-0.5, 1.0, -1.0], [0.0, 1.0, 0.5], [0.0, 0.5, 0.0], [2.0, 0.0, 0.0]))
    zero = np.zeros(3 * copies)
    off = [lo, hi, zero, zero, zero, zero]
    ref = O.stencil_solve(case, diag, off, b, solver="bicgstab", jacobi=False, rel_tol=1e-10,
                          max_iterations=50)
    assert ref.status == "Converged" and ref.restarts == 1
    got = CsrSolver(ctx).solve(*_csr(diag, off, n), b, LinearSolverSettings(
        type="bicgstab", preconditioner="none", absolute_tolerance=0.0, relative_tolerance=1e-10,
        max_iterations=50))
    assert (got.status, got.restarts, got.iterations) == (ref.status, ref.restarts, ref.iterations)
    # (the last residual is rounding: compared up to it)
    np.testing.assert_allclose(got.residual_history[:-1], ref.history[:-1], rtol=1e-8)
    assert _rel(got.solution, ref.solution) <= 1e-10
