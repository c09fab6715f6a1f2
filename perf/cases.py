"""The work that users of cfdb give it, as measurable cases.

Kinds of case (the field ``kind``):

* ``solve``: one isolated p' solve on device vectors (``POperator.solve_device``).  ``method``
  selects the FP64 Jacobi-PCG (``jacobi``), the mixed-precision one (``fp32_refined``) or the
  learned preconditioner (``learned_mg``); ``coeff`` the uniform operator or SIMPLE-like face
  coefficients; ``pinned`` a closed domain's system (reference cell pinned) or one with an
  outlet (Dirichlet patch).
* ``simple``: a stretch of outer iterations of a SIMPLE session on one cavity or duct
  (``Simple.set_state`` and ``Simple.iterate``), host fields in and out.
* ``batch``: a stretch of outer iterations of many uneven cavity and channel cases together
  (``Batch``).
* ``csr``: one solve of the reference's host CSR ``LinearSystem`` (``CsrSolver.solve``), the
  call the drop-in's linear solvers make: the BiCGSTAB momentum system.
* ``train``: one gradient step of the learned preconditioner's training
  (``POperator.mg_loss_grad``), error fields in, loss and gradient out.

Right-hand sides are sums of random-phase sinusoids with amplitude |k|^-2 (the spectrum of the
benchmark's synthetic p' systems), face coefficients follow smooth log-normal response fields
(the momentum response of a flow).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cfdapp_b200 import cfdb


def _tolerance(method, pinned):
    """The default relative tolerance of LinearSolverSettings, 1e-10.  The one pinned cell of a
    closed domain leaves the constant mode of p' nearly free: an answer that is to be the
    system's own solution, and not one of the many that meet 1e-10, is asked for at 1e-12 (the
    FP64 Jacobi-CG has that mode settled long before)."""
    return 1e-12 if pinned and method != "jacobi" else 1e-10


# ---------------------------------------------------------------- the cases

def _solve(name, dim, n, method, coeff, pinned=True):
    n = tuple(n) + (1,) * (3 - len(n))
    return {"name": name, "kind": "solve", "dim": dim, "nx": n[0], "ny": n[1], "nz": n[2],
            "method": method, "coeff": coeff, "pinned": pinned}


def listed():
    return [
        # the smallest p' systems a SIMPLE run gives to Jacobi-CG, where an iteration is pure
        # latency
        _solve("pcg_2d_40x33", 2, (40, 33), "jacobi", "faces"),
        # the reference's own method (FP64 Jacobi-CG) on an ordinary 3D grid
        _solve("pcg_3d_128", 3, (128, 128, 128), "jacobi", "uniform"),
        # the mixed-precision p' solve of an uneven 3D duct
        _solve("mixed_3d_96x80x64", 3, (96, 80, 64), "fp32_refined", "faces", False),
        # the p' system of the 129^2 cavity (odd rows), learned preconditioner
        _solve("learned_2d_129", 2, (129, 129), "learned_mg", "faces"),
        # the benchmark's headline sizes, learned preconditioner, with an outlet
        _solve("learned_2d_2048", 2, (2048, 2048), "learned_mg", "uniform", False),
        _solve("learned_3d_256", 3, (256, 256, 256), "learned_mg", "uniform", False),
        # a ragged 3D duct
        _solve("learned_3d_100x75x61", 3, (100, 75, 61), "learned_mg", "faces", False),
        # the 129^2 Re-100 cavity (upwind, linear flux), a stretch of its outer iterations
        {"name": "simple_2d_129", "kind": "simple", "flow": "cavity", "dim": 2, "nx": 129,
         "ny": 129, "nz": 1, "scheme": "upwind", "flux": "linear", "re": 100.0,
         "method": "learned_mg", "outer": 10},
        # a 3D duct with the discretization of the large runs (linear upwind, Rhie-Chow)
        {"name": "simple_3d_80x48x48", "kind": "simple", "flow": "duct", "dim": 3, "nx": 80,
         "ny": 48, "nz": 48, "scheme": "linear_upwind", "flux": "rhie_chow", "re": 100.0,
         "method": "learned_mg", "outer": 5},
        # uneven cases advanced together, every p' system by the batch's own team CG
        {"name": "batch_2d_12", "kind": "batch", "count": 12, "max_side": 256,
         "method": "jacobi", "outer": 1},
        # a momentum system handed over as host CSR arrays by the drop-in
        {"name": "csr_2d_300x200", "kind": "csr", "dim": 2, "nx": 300, "ny": 200, "nz": 1},
        # one training step at the shipped recipe's 2D grid and sample count
        {"name": "train_2d_128", "kind": "train", "dim": 2, "nx": 128, "ny": 128, "nz": 1,
         "samples": 8},
    ]


def draw(rng):
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def sides(dim, lo, hi):
        """Sides within a factor of about two of each other."""
        m = side(lo, hi)
        return tuple(max(lo, min(hi, int(round(m * rng.uniform(0.6, 1.0)))))
                     for _ in range(dim)) + (1,) * (3 - dim)

    kind = rng.choice(["jacobi", "jacobi", "fp32_refined", "learned_mg", "learned_mg",
                       "learned_mg", "simple", "simple", "batch", "csr", "train"])
    dim = rng.choice([2, 3])
    if kind in ("jacobi", "fp32_refined", "learned_mg"):
        lo, hi = {("jacobi", 2): (24, 640), ("jacobi", 3): (12, 128),
                  ("fp32_refined", 2): (24, 320), ("fp32_refined", 3): (12, 128),
                  ("learned_mg", 2): (32, 2048), ("learned_mg", 3): (16, 256)}[(kind, dim)]
        n = sides(dim, lo, hi)
        # per-face host arrays are not made for the very largest grids
        coeff = "uniform" if n[0] * n[1] * n[2] > 1_200_000 else rng.choice(["faces", "uniform"])
        # closed domains: any Jacobi-CG system; the others up to the sizes at which 1e-12 is
        # above the rounding floor of the FP64 residual
        closed = kind == "jacobi" or (dim == 2 and max(n) <= 512)
        pinned = closed and rng.random() < 0.7
        c = _solve(None, dim, n, kind, coeff, pinned)
        del c["name"]
        return c
    if kind == "simple":
        n = sides(dim, 24, 256) if dim == 2 else sides(dim, 12, 72)
        scheme = rng.choice(["upwind", "central", "linear_upwind", "quick"])
        flow = rng.choice(["cavity", "duct"])
        method = rng.choice(["learned_mg", "learned_mg", "jacobi"])
        if dim == 3 and flow == "cavity":
            method = "jacobi"
        return {"kind": "simple", "flow": flow, "dim": dim, "nx": n[0], "ny": n[1], "nz": n[2],
                "scheme": scheme, "flux": rng.choice(["linear", "rhie_chow"]),
                "re": float(rng.choice([100.0, 400.0, 1000.0]) if flow == "cavity" else 100.0),
                "method": method, "outer": rng.randint(3, 10)}
    if kind == "batch":
        return {"kind": "batch", "count": rng.randint(4, 16),
                "max_side": rng.choice([96, 128, 192, 256]),
                "method": rng.choice(["jacobi", "learned_mg"]), "outer": rng.randint(1, 2)}
    if kind == "csr":
        n = sides(dim, 24, 400) if dim == 2 else sides(dim, 12, 56)
        return {"kind": "csr", "dim": dim, "nx": n[0], "ny": n[1], "nz": n[2]}
    n = sides(dim, 48, 192) if dim == 2 else sides(dim, 16, 40)
    return {"kind": "train", "dim": dim, "nx": n[0], "ny": n[1], "nz": n[2],
            "samples": rng.randint(2, 8)}


# ------------------------------------------------------------------- inputs

def _dims(case):
    return (case["nx"], case["ny"], case["nz"])[: case["dim"]]


def _sinusoids(n, seed, count=32, waves=None):
    """A sum of random-phase cosines with amplitude |k|^-2 on the cell centres of a grid with
    n = (nx, ny[, nz]) cells, in cell order, on the GPU."""
    g = np.random.default_rng(seed)
    out = torch.zeros(tuple(reversed(n)), dtype=torch.float64, device="cuda")
    axes = [((torch.arange(m, dtype=torch.float64, device="cuda") + 0.5) / m) for m in n]
    for _ in range(count):
        k = [int(g.integers(1, max(2, min(waves or 64, m // 4) + 1))) for m in n]
        amp = 1.0 / sum(q * q for q in k)
        term = None
        for a, m in enumerate(n):
            c = torch.cos(2.0 * math.pi * (k[a] * axes[a] + float(g.uniform())))
            c = c.reshape([-1 if d == len(n) - 1 - a else 1 for d in range(len(n))])
            term = c if term is None else term * c
        out += amp * term
    return out


def _face_arrays(case, seed):
    """D_f of a smooth log-normal response on unit-spaced cells, one array per axis in
    (z,) y, x order; without a pinned cell the x-high patch is Dirichlet."""
    n = _dims(case)
    dim = case["dim"]
    if case.get("coeff") == "uniform":
        d = torch.ones(tuple(reversed(n)), dtype=torch.float64, device="cuda")
    else:
        f = _sinusoids(n, seed + 7919, count=6, waves=3)
        d = torch.exp(0.6 * f / f.abs().max())
    faces = []
    for a in range(dim):
        ax = dim - 1 - a
        m = n[a]
        inner = 0.5 * (d.narrow(ax, 1, m - 1) + d.narrow(ax, 0, m - 1))
        shape = list(d.shape)
        shape[ax] = m + 1
        f = torch.zeros(shape, dtype=torch.float64, device="cuda")
        f.narrow(ax, 1, m - 1).copy_(inner)
        if a == 0 and not case.get("pinned", True):
            f.narrow(ax, m, 1).copy_(2.0 * d.narrow(ax, m - 1, 1))
        faces.append(f)
    return faces


def _global_faces(faces):
    return torch.cat([f.reshape(-1) for f in faces]).cpu().numpy()


def _pprime_rhs(case, seed):
    """Zero-mean where the system is pinned, b[0] = 0 there (the pinned reference cell)."""
    b = _sinusoids(_dims(case), seed).reshape(-1)
    if case["pinned"]:
        b = b - b.mean()
        b[0] = 0.0
    return b.contiguous()


def _settings(method, pinned):
    return cfdb.LinearSolverSettings(
        absolute_tolerance=0.0, relative_tolerance=_tolerance(method, pinned),
        max_iterations=200000,
        preconditioner="learned_mg" if method == "learned_mg" else "jacobi",
        precision="fp32_refined" if method == "fp32_refined" else "fp64")


def _prepare_solve(case, seed):
    stream = torch.cuda.Stream()
    ctx = cfdb.Context(0, stream=stream.cuda_stream)
    n = _dims(case)
    if case["coeff"] == "uniform":
        # unit spacing, as the face form has it (the solution's scale differs otherwise)
        op = cfdb.POperator(ctx, case["dim"], n, tuple(float(m) for m in n) + (1.0,) * (3 - len(n)),
                            pinned=case["pinned"],
                            dirichlet_patch_mask=0 if case["pinned"] else 2)
    else:
        op = cfdb.POperator(ctx, case["dim"], n, face_coeff=_global_faces(_face_arrays(case, seed)),
                            pinned=case["pinned"])
    b = _pprime_rhs(case, seed)
    torch.cuda.synchronize()
    return {"kind": "solve", "op": op, "b": b, "x": torch.zeros_like(b), "stream": stream,
            "settings": _settings(case["method"], case["pinned"])}


def _flow(n, seed, through):
    """A developing flow's fields (host arrays): smooth velocities, about a unit stream along x
    when `through`, and a pressure."""
    f = [(_sinusoids(n, seed + 31 * q, count=8, waves=4)).reshape(-1) for q in range(len(n) + 1)]
    f = [0.3 * v / v.abs().max() for v in f]
    if through:
        f[0] = f[0] + 1.0
    u = [v.cpu().numpy() for v in f[:-1]]
    return u + [np.zeros_like(u[0])] * (3 - len(n)), 0.1 * f[-1].cpu().numpy()


def _bicgstab():
    return cfdb.LinearSolverSettings(absolute_tolerance=1e-12, relative_tolerance=1e-10,
                                     max_iterations=2000, type="bicgstab", preconditioner="none")


def _simple_settings(case, pinned):
    # no run of a few outer iterations meets these tolerances: every pass does all of them
    return cfdb.SIMPLESettings(max_iterations=case["outer"], velocity_tolerance=1e-9,
                               pressure_tolerance=1e-9, continuity_tolerance=1e-9,
                               convection_scheme=case.get("scheme", "upwind"),
                               face_flux=case.get("flux", "linear"),
                               momentum_solver=_bicgstab(),
                               pressure_solver=_settings(case["method"], pinned))


def _prepare_simple(case, seed):
    n = _dims(case)
    vbc = [("wall", (0.0, 0.0, 0.0))] * (2 * len(n))
    pbc = [("fixed_gradient", 0.0)] * (2 * len(n))
    closed = case["flow"] == "cavity"
    if closed:
        vbc[3] = ("moving_wall", (1.0, 0.0, 0.0))
    else:
        vbc[0], vbc[1] = ("inlet", (1.0, 0.0, 0.0)), ("outlet", (0.0, 0.0, 0.0))
        pbc[1] = ("fixed_value", 0.0)
    length = tuple(m / min(n) for m in n) + (1.0,) * (3 - len(n))  # equal spacings
    sc = cfdb.SimpleCase(len(n), n, length, tuple(vbc), tuple(pbc), 1.0, 1.0 / case["re"])
    ctx = cfdb.Context(0)
    return {"kind": "simple", "session": cfdb.Simple(ctx, sc, _simple_settings(case, closed)),
            "fields": _flow(n, seed, not closed), "outer": case["outer"]}


def _batch_grids(case):
    """(nx, ny) of every case: square cavities, and every third one a 2:1 channel."""
    sides = [s for s in (48, 64, 96, 128, 192, 256) if s <= case["max_side"]]
    got = [sides[-1 - (q * q + q) // 2 % len(sides)] for q in range(case["count"])]
    return [(s, s // 2 if q % 3 == 2 else s) for q, s in enumerate(got)]


def _prepare_batch(case, seed):
    g = np.random.default_rng(seed)
    cases = []
    for nx, ny in _batch_grids(case):
        mu = 1.0 / float(g.uniform(100.0, 1000.0))
        cases.append(cfdb.SimpleCase.cavity(2, nx, mu=mu) if nx == ny else
                     cfdb.SimpleCase.channel(nx, ny, 2.0, 1.0, mu=10.0 * mu))
    ctx = cfdb.Context(0)
    fields = [_flow(c.n, seed + 101 * q, c.n[0] != c.n[1]) for q, c in enumerate(cases)]
    return {"kind": "batch", "batch": cfdb.Batch(ctx, cases, _simple_settings(case, True)),
            "fields": fields, "outer": case["outer"]}


def _momentum_bands(case, seed):
    """Diagonal and couplings [(axis, side)] of an upwind momentum system with implicit
    under-relaxation 0.7 in a smooth flow, and its right-hand side."""
    n = _dims(case)
    dim = len(n)
    shape = tuple(reversed(n))
    vel = [_sinusoids(n, seed + 31 * a, count=8, waves=4) for a in range(dim)]
    diff = 0.05
    off = {}
    diag = torch.zeros(shape, dtype=torch.float64, device="cuda")
    for a in range(dim):
        ax = dim - 1 - a
        v = vel[a] / vel[a].abs().max()
        f = 0.5 * (v.narrow(ax, 1, n[a] - 1) + v.narrow(ax, 0, n[a] - 1))  # flux of inner faces
        lo = torch.zeros_like(diag)
        hi = torch.zeros_like(diag)
        lo.narrow(ax, 1, n[a] - 1).copy_(-(diff + torch.clamp(f, min=0.0)))
        hi.narrow(ax, 0, n[a] - 1).copy_(-(diff + torch.clamp(-f, min=0.0)))
        off[(a, 0)], off[(a, 1)] = lo, hi
        diag -= lo + hi
    diag = (diag + 0.02) / 0.7
    b = _sinusoids(n, seed + 997, count=16)
    return diag, off, b


def _csr_of(diag, off, n):
    """The reference's CSR arrays (ascending columns) of the banded system, as host arrays."""
    dim = len(n)
    stride = [1, n[0], n[0] * (n[1] if dim > 1 else 1)]
    cells = int(np.prod(n))
    idx = np.arange(cells).reshape(tuple(reversed(n)))
    cols, vals, keep = [], [], []
    order = [(a, 0) for a in reversed(range(dim))] + [None] + [(a, 1) for a in range(dim)]
    for o in order:
        if o is None:
            cols.append(idx.ravel())
            vals.append(diag.cpu().numpy().ravel())
            keep.append(np.ones(cells, dtype=bool))
            continue
        a, s = o
        pos = np.arange(n[a]).reshape([-1 if d == dim - 1 - a else 1 for d in range(dim)])
        inside = np.broadcast_to(pos > 0 if s == 0 else pos < n[a] - 1, idx.shape)
        cols.append((idx + (stride[a] if s else -stride[a])).ravel())
        vals.append(off[o].cpu().numpy().ravel())
        keep.append(inside.ravel())
    cols, vals, keep = (np.stack(v, axis=1) for v in (cols, vals, keep))
    offsets = np.concatenate([[0], np.cumsum(keep.sum(axis=1))]).astype(np.uint64)
    return offsets, cols[keep].astype(np.uint64), vals[keep]


def _prepare_csr(case, seed):
    diag, off, b = _momentum_bands(case, seed)
    ro, ci, v = _csr_of(diag, off, _dims(case))
    ctx = cfdb.Context(0)
    return {"kind": "csr", "solver": cfdb.CsrSolver(ctx), "settings": _bicgstab(),
            "system": (ro, ci, v, b.reshape(-1).cpu().numpy())}


def _error_fields(case, seed):
    """Unit-RMS error fields with content at every scale (host float32, the training input)."""
    n = _dims(case)
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = tuple(reversed(n))
    out = torch.zeros((case["samples"],) + shape, dtype=torch.float64, device="cuda")
    level = 0
    while True:
        f = 2 ** level
        cs = [(m + f - 1) // f for m in shape]
        if min(cs) < 2:
            break
        up = torch.randn([case["samples"]] + cs, generator=g, dtype=torch.float64, device="cuda")
        for ax in range(len(shape)):
            up = up.repeat_interleave(f, dim=1 + ax)
        out += up[(slice(None),) + tuple(slice(0, m) for m in shape)] * (1.5 ** level)
        level += 1
    out = out.reshape(case["samples"], -1)
    return (out / out.square().mean(dim=1, keepdim=True).sqrt()).float().cpu().numpy()


def _prepare_train(case, seed):
    ctx = cfdb.Context(0)
    op = cfdb.POperator(ctx, case["dim"], _dims(case),
                        face_coeff=_global_faces(_face_arrays(case, seed)))
    return {"kind": "train", "op": op, "errors": _error_fields(case, seed)}


def prepare(case, seed):
    return {"solve": _prepare_solve, "simple": _prepare_simple, "batch": _prepare_batch,
            "csr": _prepare_csr, "train": _prepare_train}[case["kind"]](case, seed)


# --------------------------------------------------------------------- runs

def run(state):
    kind = state["kind"]
    if kind == "solve":
        with torch.cuda.stream(state["stream"]):
            x = state["x"].zero_()
        state["op"].solve_device(state["b"].data_ptr(), x.data_ptr(), state["settings"])
        return {"x": x}
    if kind == "simple":
        (u, v, w), p = state["fields"]
        s = state["session"]
        s.set_state(u, v, w, p)
        r = s.iterate(state["outer"])
        return {"u": r.u, "v": r.v, "w": r.w, "p": r.p, "flux": r.flux}
    if kind == "batch":
        b = state["batch"]
        for k, ((u, v, w), p) in enumerate(state["fields"]):
            b.set_state(k, u, v, w, p)
        b.iterate(state["outer"])
        got = [b.get_state(k) for k in range(len(state["fields"]))]
        return {name: np.concatenate([g[q] for g in got])
                for q, name in ((0, "u"), (1, "v"), (3, "p"), (4, "flux"))}
    if kind == "csr":
        return {"x": state["solver"].solve(*state["system"], state["settings"],
                                           history_cap=0).solution}
    loss, gk, gc = state["op"].mg_loss_grad(state["errors"])
    # the trainer's weights are float32 (what cfdb_mg_set_weights takes), and so is its step
    return {"loss": np.float32(loss), "kernels": gk.astype(np.float32),
            "coarse": gc.astype(np.float32)}


def work(case):
    """What a pass cannot do without: the input fields read once and the results written once;
    for a solve also the flops of one application of the operator."""
    if case["kind"] == "batch":
        cells = sum(nx * ny for nx, ny in _batch_grids(case))
        dim = 2
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
        dim = case["dim"]
    flops = (4.0 * dim + 1.0) * cells
    if case["kind"] == "solve":
        faces = dim if case["coeff"] == "faces" else 0
        return {"bytes": 8.0 * cells * (2 + faces), "flops": flops}
    if case["kind"] in ("simple", "batch"):
        # velocities and pressure in and out, the face fluxes out
        return {"bytes": 8.0 * cells * (2 * (dim + 1) + dim), "flops": case["outer"] * flops}
    if case["kind"] == "csr":
        nnz = cells * (2 * dim + 1)
        return {"bytes": 16.0 * nnz + 8.0 * cells * 3, "flops": 2.0 * nnz}
    # the error fields and the operator's faces in; forward and backward passes of a 3^dim kernel
    return {"bytes": 4.0 * cells * case["samples"] + 8.0 * cells * dim,
            "flops": case["samples"] * cells * (4.0 * 3 ** dim + 2 * flops / cells)}


# ------------------------------------------------------- values in 64 bits

def _apply_faces(faces, x):
    y = torch.zeros_like(x)
    dim = x.dim()
    for a, f in enumerate(faces):
        ax = dim - 1 - a
        m = x.shape[ax]
        y += (f.narrow(ax, 0, m) + f.narrow(ax, 1, m)) * x
        inner = f.narrow(ax, 1, m - 1)
        y.narrow(ax, 1, m - 1).sub_(inner * x.narrow(ax, 0, m - 1))
        y.narrow(ax, 0, m - 1).sub_(inner * x.narrow(ax, 1, m - 1))
    return y


def _cosine_solve(r, mean):
    """Inverse of the uniform Neumann Laplacian (unit coupling, scaled by `mean`) on the
    zero-mean fields, by even extension and FFT."""
    y = r
    axes = list(range(r.dim()))
    for ax in axes:
        y = torch.cat([y, y.flip(ax)], dim=ax)
    y = torch.fft.rfftn(y)
    eig = torch.zeros(y.shape, dtype=torch.float64, device=r.device)
    for ax in axes:
        m = 2 * r.shape[ax]
        k = torch.arange(y.shape[ax], dtype=torch.float64, device=r.device)
        s = 4.0 * torch.sin(math.pi * k / m) ** 2
        eig += s.reshape([-1 if d == ax else 1 for d in axes])
    zero = (0,) * r.dim()
    eig[zero] = 1.0
    y = y / (mean * eig)
    y[zero] = 0.0
    y = torch.fft.irfftn(y, s=[2 * m for m in r.shape])
    return y[tuple(slice(0, m) for m in r.shape)]


def _exact_solve(case, seed):
    """Preconditioned CG to rounding on the singular Neumann form (pinned: all rows but the
    reference cell's are the pinned system's, and the solution is shifted to x[0] = b[0]) or on
    the Dirichlet system."""
    faces = _face_arrays(case, seed)
    dim = case["dim"]
    b = _pprime_rhs(case, seed).reshape(tuple(reversed(_dims(case))))
    pinned = case["pinned"]
    rhs = b.clone()
    if pinned:
        rhs[(0,) * dim] = -(b.sum() - b[(0,) * dim])
    mean = float(sum(f.sum() / f.numel() for f in faces) / dim)
    dirichlet = 0.0 if pinned else 1.0

    def precondition(r):
        z = _cosine_solve(r - r.mean(), mean)
        # the constant mode of the Dirichlet system, from its own Rayleigh quotient
        return z + dirichlet * r.mean() / mode

    mode = 1.0 if pinned else float(_apply_faces(faces, torch.ones_like(b)).mean())
    x = torch.zeros_like(b)
    for _ in range(3):  # restarted on the true residual
        r = rhs - _apply_faces(faces, x)
        first = float(r.norm())
        if first <= 1e-17 * float(rhs.norm()):
            break
        z = precondition(r)
        p, rz = z.clone(), float((r * z).sum())
        for _ in range(400):
            q = _apply_faces(faces, p)
            pq = float((p * q).sum())
            if not rz > 0.0 or not pq > 0.0:  # nothing but rounding is left
                break
            alpha = rz / pq
            x = x + alpha * p
            r = r - alpha * q
            if float(r.norm()) <= 1e-9 * first:
                break
            z = precondition(r)
            new = float((r * z).sum())
            p, rz = z + (new / rz) * p, new
    if pinned:
        x = x - x[(0,) * dim] + b[(0,) * dim]
    return {"x": x.reshape(-1)}


def _exact_csr(case, seed):
    """The relaxed system is diagonally dominant by 1/0.7, so Jacobi's iteration gains a digit
    every seven sweeps."""
    diag, off, b = _momentum_bands(case, seed)
    n = _dims(case)
    x = torch.zeros_like(b)
    for _ in range(160):
        s = b.clone()
        for (a, side), o in off.items():
            ax = len(n) - 1 - a
            m = n[a]
            if side == 0:
                s.narrow(ax, 1, m - 1).sub_(o.narrow(ax, 1, m - 1) * x.narrow(ax, 0, m - 1))
            else:
                s.narrow(ax, 0, m - 1).sub_(o.narrow(ax, 0, m - 1) * x.narrow(ax, 1, m - 1))
        x = s / diag
    return {"x": x.reshape(-1).cpu().numpy()}


def _pairs(x, axes):
    """Sums of adjacent pairs along `axes` (odd extents padded with zeros)."""
    for ax in axes:
        m = x.shape[ax]
        if m % 2:
            pad = list(x.shape)
            pad[ax] = 1
            x = torch.cat([x, x.new_zeros(pad)], dim=ax)
        x = x.unflatten(ax, (-1, 2)).sum(dim=ax + 1)
    return x


def _exact_train(case, seed):
    """The V-cycle network and its loss in plain torch at 64 bits, the gradient by autograd."""
    dim = case["dim"]
    w = _shipped_weights(dim)
    kernels = torch.tensor(w["kernels"], dtype=torch.float64, device="cuda", requires_grad=True)
    coarse = torch.tensor(w["coarse_weights"], dtype=torch.float64, device="cuda",
                          requires_grad=True)
    levels = [_face_arrays(case, seed)]
    while True:
        f = levels[-1]
        n = [f[a].shape[dim - 1 - a] - 1 for a in range(dim)]
        if len(levels) > 1 and (min(n) <= 4 or math.prod(n) <= 64):
            break
        nxt = []
        for a in range(dim):
            ax = dim - 1 - a
            m = n[a]
            pos = torch.tensor([min(2 * q, m) for q in range((m + 1) // 2 + 1)], device="cuda")
            nxt.append(_pairs(f[a].index_select(ax, pos), [d for d in range(dim) if d != ax]))
        levels.append(nxt)

    def lap(l, x):  # a leading sample axis
        y = torch.zeros_like(x)
        for a, f in enumerate(levels[l]):
            ax = dim - 1 - a
            m = x.shape[1 + ax]
            y = y + (f.narrow(ax, 0, m) + f.narrow(ax, 1, m)) * x
            inner = f.narrow(ax, 1, m - 1)
            shape = list(x.shape)
            shape[1 + ax] = 1
            z = x.new_zeros(shape)
            y = y - torch.cat([z, inner * x.narrow(1 + ax, 0, m - 1)], dim=1 + ax)
            y = y - torch.cat([inner * x.narrow(1 + ax, 1, m - 1), z], dim=1 + ax)
        return y

    def scale(l):
        d = 0.0
        for a, f in enumerate(levels[l]):
            ax = dim - 1 - a
            m = f.shape[ax] - 1
            d = d + f.narrow(ax, 0, m) + f.narrow(ax, 1, m)
        return torch.rsqrt(d)

    def conv(l, u):
        k = kernels[min(l, len(kernels) - 1)]
        k = k[9:18].reshape(3, 3) if dim == 2 else k.reshape(3, 3, 3)
        fn = torch.nn.functional.conv2d if dim == 2 else torch.nn.functional.conv3d
        return fn(u[:, None], k[None, None], padding=1)[:, 0]

    def cycle(l, r):
        s = scale(l)
        if l == len(levels) - 1:
            x = torch.zeros_like(r)
            for _ in range(w["coarse_sweeps"]):
                x = x + 0.8 * s * s * (r - lap(l, x))
            return x
        x = s * conv(l, s * r)
        for _ in range(w["nu"] - 1):
            x = x + s * conv(l, s * (r - lap(l, x)))
        e = cycle(l + 1, _pairs(r - lap(l, x), range(1, dim + 1)))
        for ax in range(1, dim + 1):
            e = e.repeat_interleave(2, dim=ax).narrow(ax, 0, r.shape[ax])
        x = x + coarse[min(l, len(coarse) - 1)] * e
        for _ in range(w["nu"]):
            x = x + s * conv(l, s * (r - lap(l, x)))
        return x

    e = torch.from_numpy(_error_fields(case, seed)).cuda().double()
    mask = torch.ones(e.shape[1], dtype=torch.float64, device="cuda")
    mask[0] = 0.0  # the pinned reference cell
    shape = (len(e),) + tuple(reversed(_dims(case)))
    e, mask = (e * mask).reshape(shape), mask.reshape(shape[1:])
    z = cycle(0, lap(0, e) * mask) * mask
    d = z - e
    axes = list(range(1, dim + 1))
    loss = ((d * lap(0, d)).sum(dim=axes) / (e * lap(0, e)).sum(dim=axes)).mean()
    loss.backward()
    gk = np.zeros((cfdb.MG_MAX_LEVELS, cfdb.MG_TAPS))
    gc = np.zeros(cfdb.MG_MAX_LEVELS)
    g = kernels.grad.cpu().numpy()
    # a tap and its mirror image are one weight: both carry the sum of their gradients
    g = g + g[:, ::-1] * (np.arange(cfdb.MG_TAPS) != 13)
    gk[: len(g)] = g
    gc[: len(coarse)] = coarse.grad.cpu().numpy()
    return {"loss": np.float64(loss.item()), "kernels": gk, "coarse": gc}


def _shipped_weights(dim):
    """The shipped weight set, as a program reads it back from its context."""
    with cfdb.Context(0) as ctx:
        return ctx.mg_get_weights(dim)


def exact(case, seed):
    if case["kind"] == "solve":
        return _exact_solve(case, seed)
    if case["kind"] == "csr":
        return _exact_csr(case, seed)
    if case["kind"] == "train":
        return _exact_train(case, seed)
    return None  # a stretch of a nonlinear iteration
