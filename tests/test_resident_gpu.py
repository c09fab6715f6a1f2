"""The on-chip Krylov solves (resident.cuh) against the CPU oracle at the edges
of their dispatch: one block, whole and partial blocks of a cluster, the
cluster's largest system and the first of the grid team's, both thread counts
of the grid team, and planes too large to be kept in shared memory.

Both sides run the same method with the same arithmetic up to the order of the
sums, so after a fixed number of iterations the iterates agree to rounding
(1e-10 relative L2, the bound of the FP64 parity tests being 1e-9).
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

GRIDS = [(2, 2), (23, 22), (32, 16), (31, 33), (129, 63), (192, 192), (193, 192), (700, 433),
         (703, 433), (7, 5, 3), (33, 33, 33), (200, 190, 3), (61, 43, 40)]


def _system(n, seed, outlet):
    """A SIMPLE-like p' system with variable face coefficients."""
    dim = len(n)
    pbc = [("fixed_gradient", 0.0)] * (2 * dim)
    vbc = [("wall", (0, 0, 0))] * (2 * dim)
    if outlet:
        pbc[1] = ("fixed_value", 0.0)
        vbc[0], vbc[1] = ("inlet", (1.0, 0, 0)), ("outlet", (0, 0, 0))
    case = O.Case(dim, n, tuple(float(m) for m in n), vbc, pbc)
    rng = np.random.default_rng(seed)
    d = [rng.uniform(0.5, 2.0, case.cells()) for _ in range(3)]
    flux = rng.normal(size=case.faces())
    return (case,) + O.assemble_pprime(case, 1.0, flux, *d)


def _rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("n", GRIDS)
def test_pcg_iterates_match_oracle(ctx, n):
    from cfdapp_b200.cfdb import LinearSolverSettings, POperator
    for outlet in (False, True):
        case, fc, diag, off, rhs = _system(n, 5, outlet)
        x0 = np.random.default_rng(6).normal(size=case.cells())
        its = min(40, case.cells() // 4)
        ref = O.stencil_solve(case, diag, off, rhs, x0=x0, rel_tol=1e-30, max_iterations=its)
        op = POperator(ctx, len(n), n, tuple(float(m) for m in n), face_coeff=fc,
                       pinned=not outlet)
        got = op.solve(rhs, LinearSolverSettings(absolute_tolerance=0.0, relative_tolerance=1e-30,
                                                 max_iterations=its), x0=x0)
        assert got.status == ref.status and got.iterations == ref.iterations
        np.testing.assert_allclose(got.residual_history, ref.history, rtol=1e-8)
        assert _rel(got.solution, ref.solution) <= 1e-10


@pytest.mark.parametrize("n", [(40, 33), (193, 192), (17, 19, 23), (64, 50, 40)])
def test_pcg_of_the_uniform_operator_matches_its_face_form(ctx, n):
    """Per-axis tables against the same coefficients as face arrays."""
    from cfdapp_b200.cfdb import LinearSolverSettings, POperator
    dim = len(n)
    length = tuple(float(m) for m in n)
    case = O.Case(dim, n, length, [("wall", (0, 0, 0))] * (2 * dim),
                  [("fixed_gradient", 0.0)] * (2 * dim))
    ones = np.ones(case.cells())
    fc, _, _, _ = O.assemble_pprime(case, 1.0, np.zeros(case.faces()), ones, ones, ones)
    b = np.random.default_rng(2).normal(size=case.cells())
    s = LinearSolverSettings(absolute_tolerance=0.0, relative_tolerance=1e-30, max_iterations=50)
    tab = POperator(ctx, dim, n, length).solve(b, s)
    arr = POperator(ctx, dim, n, length, face_coeff=fc).solve(b, s)
    np.testing.assert_allclose(tab.residual_history, arr.residual_history, rtol=1e-12)
    assert _rel(tab.solution, arr.solution) <= 1e-13


def _csr(diag, off, n):
    """The rows of a banded system in the reference's column order (host CSR arrays)."""
    dim = len(n)
    stride = [1, n[0], n[0] * n[1]]
    idx = np.arange(int(np.prod(n)))
    pos = [(idx // stride[a]) % n[a] for a in range(dim)]
    cols, vals, keep = [], [], []
    order = [(a, 0) for a in reversed(range(dim))] + [None] + [(a, 1) for a in range(dim)]
    for o in order:
        if o is None:
            c, v, k = idx, diag, np.ones(len(idx), bool)
        else:
            a, s = o
            c, v = idx + (stride[a] if s else -stride[a]), off[2 * a + s]
            k = pos[a] < n[a] - 1 if s else pos[a] > 0
        cols.append(c)
        vals.append(v)
        keep.append(k)
    cols, vals, keep = (np.stack(q, axis=1) for q in (cols, vals, keep))
    ro = np.concatenate([[0], np.cumsum(keep.sum(axis=1))])
    return ro, cols[keep], vals[keep]


@pytest.mark.parametrize("n", GRIDS)
@pytest.mark.parametrize("method", ["bicgstab", "cg"])
@pytest.mark.parametrize("jacobi", [False, True])
def test_band_solves_match_oracle(ctx, n, method, jacobi):
    """A diagonally dominant banded system (symmetric for CG, upwind-like for BiCGSTAB)
    through the CSR entry point."""
    from cfdapp_b200.cfdb import CsrSolver, LinearSolverSettings
    dim = len(n)
    case = O.Case(dim, n, tuple(float(m) for m in n), [("wall", (0, 0, 0))] * (2 * dim),
                  [("fixed_gradient", 0.0)] * (2 * dim))
    cells = case.cells()
    rng = np.random.default_rng(8)
    stride = [1, n[0], n[0] * n[1]]
    idx = np.arange(cells)
    off = [np.zeros(cells) for _ in range(6)]
    total = np.zeros(cells)
    for a in range(dim):
        inner = (idx // stride[a]) % n[a] < n[a] - 1
        lo_of = idx[inner]
        w = -rng.uniform(0.5, 1.5, len(lo_of))
        off[2 * a + 1][lo_of] = w
        off[2 * a][lo_of + stride[a]] = w if method == "cg" else w * rng.uniform(0.2, 1.0, len(w))
        total += np.abs(off[2 * a]) + np.abs(off[2 * a + 1])
    diag = (total + 0.05) / 0.8
    b, x0 = rng.normal(size=cells), rng.normal(size=cells)
    its = min(6, cells // 2)
    ref = O.stencil_solve(case, diag, off, b, x0=x0, solver=method, jacobi=jacobi, rel_tol=1e-30,
                          max_iterations=its)
    s = LinearSolverSettings(type=method, preconditioner="jacobi" if jacobi else "none",
                             absolute_tolerance=0.0, relative_tolerance=1e-30, max_iterations=its)
    got = CsrSolver(ctx).solve(*_csr(diag, off, n), b, s, x0=x0)
    assert got.status == ref.status and got.iterations == ref.iterations
    np.testing.assert_allclose(got.residual_history, ref.history, rtol=1e-8)
    assert _rel(got.solution, ref.solution) <= 1e-10


# grids at the edges of the learned solve's cluster form: one block with all
# planes, fewer planes than blocks, partial last blocks, odd coarsenings, the
# largest that fit, and (the last of each dimension) ones that do not
@pytest.mark.parametrize("n", [(8, 8), (17, 5), (31, 129), (129, 31), (96, 90), (255, 257), (301, 290),
                               (5, 6, 7), (9, 24, 37), (33, 33, 33), (24, 30, 9), (41, 40, 39)])
@pytest.mark.parametrize("outlet", [True, False])
def test_learned_solve_matches_jacobi(ctx, n, outlet):
    """The learned FCG and the Jacobi-CG of one system, both to a relative residual of 1e-12:
    the solutions agree within 1e-9 with an outlet (the FP64 parity bar), 1e-7 in a closed
    domain, whose nearly free constant mode the residual sees 10^4 times less."""
    from cfdapp_b200.cfdb import LinearSolverSettings, POperator
    case, fc, diag, off, rhs = _system(n, 9, outlet)
    ref_cell = 0 if outlet else case.cells() // 2
    if not outlet:
        rhs = rhs - rhs.mean()
        rhs[ref_cell] = 0.0
    op = POperator(ctx, len(n), n, tuple(float(m) for m in n), face_coeff=fc, pinned=not outlet,
                   reference_cell=ref_cell)
    got = {}
    for pc in ("jacobi", "learned_mg"):
        got[pc] = op.solve(rhs, LinearSolverSettings(absolute_tolerance=0.0, preconditioner=pc,
                                                     relative_tolerance=1e-12, max_iterations=20000))
        assert got[pc].status == "Converged"
        assert got[pc].fallback_iterations == 0
    assert got["learned_mg"].iterations <= got["jacobi"].iterations
    assert _rel(got["learned_mg"].solution, got["jacobi"].solution) <= (1e-9 if outlet else 1e-7)
