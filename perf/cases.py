"""The work a program gives this solver, as timed cases.

A case is a matrix family with its sizes, a structure ("SPD" Cholesky, "S" LDL^T, "G" LU), a precision, the
right-hand sides and one of three operations:

* ``step``: new values in the solver's pattern, factorization, solve (what a time step, a Newton step or an
  interior-point iteration does). "G" solves with A and with A^T, "S" of a KKT also reads the inertia;
* ``solve``: right-hand sides through a factor in hand;
* ``grad``: the differentiable solve, forward and backward.

``prepare`` makes the matrix, analyses it and builds the plan; ``run`` is one pass through ``DirectSolver``
(or ``UnevenBatch``, ``adjoint.solve``). The right-hand sides are A X for a random X, so the exact result is
known without solving anything: X, up to the rounding of A X (about cond(A) 1e-16, far below any tolerance here).
"""
from __future__ import annotations

import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sparsedirectsolver.jl_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from sdsb200 import adjoint, analyze_csr  # noqa: E402
from sdsb200 import matrices as M  # noqa: E402
from sdsb200.batch import UnevenBatch  # noqa: E402
from sdsb200.solver import DirectSolver  # noqa: E402


def _case(name, family, op="step", **kw):
    c = dict(name=name, family=family, op=op, structure="SPD", nx=0, ny=0, nz=0, nj=0, nrhs=1, precision="fp64",
             ir_steps=0, ir_tol=0.0, reordering="default", maxwidth=32, members=1)
    c.update(kw)
    return c


def listed():
    return [
        # one small system on its own, where launches and host work are everything
        _case("spd_lap2d_16", "lap2d", nx=16, ny=16),
        # the 64 x 64 five-point problem with the minimum-degree ordering
        _case("spd_lap2d_64", "lap2d", nx=64, ny=64, reordering="amd"),
        # the 300 x 300 five-point problem, all defaults: many small fronts, a few of middle size
        _case("spd_lap2d_300", "lap2d", nx=300, ny=300),
        # the benchmark's 48^3 seven-point problem, 4 right-hand sides, in FP64 and with an FP32 factor
        _case("spd_lap3d_48", "lap3d", nx=48, ny=48, nz=48, nrhs=4, reordering="nd", maxwidth=512),
        _case("spd_lap3d_48_mixed", "lap3d", nx=48, ny=48, nz=48, nrhs=4, reordering="nd", maxwidth=512,
              precision="fp32", ir_steps=2),
        # many right-hand sides through one factor, a ragged grid
        _case("spd_lap3d_solve13", "lap3d", op="solve", nx=41, ny=47, nz=37, nrhs=13, reordering="nd"),
        # LDL^T of a definite 3-D problem (no knowledge of definiteness), one right-hand side
        _case("sym_lap3d_40", "lap3d", structure="S", nx=40, ny=40, nz=40, reordering="nd"),
        # an interior-point KKT system: Bunch-Kaufman, refinement to a tolerance, inertia
        _case("sym_kkt_80", "kkt", structure="S", nx=80, ny=75, nj=2250, ir_steps=20, ir_tol=1e-12),
        # unsymmetric convection-diffusion, 8 right-hand sides with A and with A^T
        _case("lu_cd3d_40", "cd3d", structure="G", nx=40, ny=40, nz=40, nrhs=8, reordering="nd"),
        # a uniform batch: one pattern, 256 sets of values
        _case("batch_lap2d_96x256", "lap2d", nx=96, ny=96, members=256),
        # many unrelated small systems at once, FP32 factors with one refinement step
        _case("uneven_256_mixed", "uneven", nx=16, ny=48, members=256, precision="fp32", ir_steps=1),
        # the differentiable solve, forward and backward, a ragged unsymmetric problem
        _case("grad_cd3d_21", "cd3d", op="grad", structure="G", nx=21, ny=23, nz=19, nrhs=2, reordering="nd"),
    ]


def _log(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    """One more case of the listed ranges; every family, structure and precision, ragged sizes."""
    kind = rng.choice(["lap2d", "lap2d", "lap3d", "lap3d", "sym3d", "kkt", "cd3d", "cd3d", "batch", "uneven"])
    mixed = rng.random() < 0.35
    kw = dict(precision="fp32", ir_steps=2) if mixed else {}
    op = rng.choice(["step", "step", "step", "solve", "grad"])
    order = rng.choice(["nd", "amd", "default"])
    if kind == "lap2d":
        c = _case("", "lap2d", op, nx=_log(rng, 12, 300), ny=_log(rng, 12, 300), nrhs=rng.randint(1, 8),
                  reordering=order, **kw)
    elif kind in ("lap3d", "sym3d"):
        hi = 44 if kind == "lap3d" else 34
        c = _case("", "lap3d", op, structure="SPD" if kind == "lap3d" else "S", nx=_log(rng, 6, hi), ny=_log(rng, 6, hi),
                  nz=_log(rng, 6, hi), nrhs=rng.randint(1, 13), reordering="nd", maxwidth=rng.choice([32, 128, 512]), **kw)
    elif kind == "kkt":
        nx, ny = _log(rng, 10, 70), _log(rng, 10, 70)
        c = _case("", "kkt", "step", structure="S", nx=nx, ny=ny, nj=max(1, int(nx * ny * rng.uniform(0.1, 0.375))),
                  ir_steps=20, ir_tol=1e-12, precision="fp32" if mixed else "fp64")
    elif kind == "cd3d":
        c = _case("", "cd3d", op, structure="G", nx=_log(rng, 6, 36), ny=_log(rng, 6, 36), nz=_log(rng, 6, 36),
                  nrhs=rng.randint(1, 8), reordering="nd", **kw)
    elif kind == "batch":
        nx, ny = _log(rng, 8, 96), _log(rng, 8, 96)
        c = _case("", "lap2d", "step", nx=nx, ny=ny, members=min(256, _log(rng, 2, 256)), **kw)
    else:
        lo = rng.randint(8, 24)
        c = _case("", "uneven", "step", nx=lo, ny=rng.randint(lo, 48), members=_log(rng, 8, 256), **kw)
    if c["op"] == "grad":      # differentiation needs an accurate solution, not a refined one
        c.update(precision="fp64", ir_steps=0)
    del c["name"]
    return c


# -- inputs ----------------------------------------------------------------------------------------------------

def _congruence(A, rng, spread):
    """D A D with a random diagonal D in [1 - spread, 1 + spread]: other values, the same definiteness."""
    d = rng.uniform(1.0 - spread, 1.0 + spread, A.shape[0])
    r = np.repeat(np.arange(A.shape[0]), np.diff(A.indptr))
    A = A.copy()
    A.data = A.data * d[r] * d[A.indices]
    return A


def _matrix(c, seed):
    rng = np.random.default_rng([seed, 1])
    if c["family"] == "lap2d":
        return M.lap2d_shifted(c["nx"], c["ny"], seed=seed)
    if c["family"] == "lap3d":
        return _congruence(M.lap3d(c["nx"], c["ny"], c["nz"]), rng, 0.1)
    if c["family"] == "cd3d":
        return M.convection_diffusion3d(c["nx"], c["ny"], c["nz"], seed=seed)
    # an interior-point method keeps the pattern and rescales the values as the barrier moves
    return _congruence(M.kkt(c["nx"], c["ny"], c["nj"], seed=0), rng, 0.5)


def _systems(c, seed):
    rng = np.random.default_rng([seed, 1])
    return [_congruence(A, rng, 0.1) for A in M.uneven_batch(c["members"], c["nx"], c["ny"], 0.1, 0)]


def _size(c):
    return {"lap2d": c["nx"] * c["ny"], "kkt": c["nx"] * c["ny"] + c["nj"]}.get(c["family"], c["nx"] * c["ny"] * c["nz"])


def _uneven_size(c):
    # uneven_batch's own draw of the grid sizes
    s = np.random.default_rng(0).integers(c["nx"], c["ny"] + 1, c["members"])
    return int((s.astype(np.int64) ** 2).sum())


def _solution(c, seed, n, which=0):
    rng = np.random.default_rng([seed, 2 + which])
    shape = (c["members"], n) if c["family"] == "lap2d" and c["members"] > 1 else (n,) if c["nrhs"] == 1 else (n, c["nrhs"])
    return rng.uniform(-1.0, 1.0, shape)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _params(c):
    p = dict(max_nrhs=min(8, c["nrhs"]), reordering_alg=c["reordering"], amalgamation=(c["maxwidth"], 0.25, 8),
             ir_n_steps=c["ir_steps"], ir_tol=c["ir_tol"])
    if c["nrhs"] > 8:
        p["max_nrhs"] = c["nrhs"]
    if c["precision"] == "fp32":
        p["factor_precision"] = "fp32"
    if c["structure"] == "G":
        p["pivot_threshold"] = 0.1
    return p


def prepare(case, seed):
    c = case
    if c["family"] == "uneven":
        ub = UnevenBatch(_systems(c, seed), c["structure"], **_params(c))
        ub.execute("analysis")
        A = ub.A
        return dict(case=c, solver=ub, values=_dev(A.data), b=_dev(A @ _solution(c, seed, A.shape[0])))
    A = _matrix(c, seed)
    n = A.shape[0]
    X = _solution(c, seed, n)
    if X.ndim == 2 and c["members"] > 1:      # uniform batch: member k is D_k A D_k
        vals = M.batch_members(A, c["members"], spread=0.1, seed=seed)
        r = np.repeat(np.arange(n), np.diff(A.indptr))
        b = np.stack([np.bincount(r, v * x[A.indices], n) for v, x in zip(vals, X)])
        ds = DirectSolver((A.indptr, A.indices, vals.reshape(-1), n), c["structure"], **_params(c))
        ds.execute("analysis")
        return dict(case=c, solver=ds, values=_dev(vals.reshape(-1)), b=_dev(b))
    ds = DirectSolver(A, c["structure"], **_params(c))
    ds.execute("analysis")
    s = dict(case=c, solver=ds, values=_dev(A.data), b=_dev(A @ X))
    if c["structure"] == "G":
        s["bt"] = _dev(A.T @ _solution(c, seed, n, 1))
    if c["op"] == "solve":
        ds.execute("factorization")
    if c["op"] == "grad":
        # the loss's derivative A^T Y gives b-bar = Y (the symmetric structures' too)
        s["xbar"] = _dev(A.T @ _solution(c, seed, n, 1))
        s["values"].requires_grad_()
        s["b"].requires_grad_()
    return s


def run(state):
    c, ds, b = state["case"], state["solver"], state["b"]
    if c["op"] == "grad":
        x = adjoint.solve(ds, state["values"], b)
        abar, bbar = torch.autograd.grad(x, (state["values"], b), state["xbar"])
        return {"x": x.detach(), "abar": abar, "bbar": bbar}
    out = {}
    if c["op"] == "step":
        if c["family"] == "uneven":
            ds.solver.update(state["values"])
            out["info"] = ds.execute("factorization")
        else:
            ds.update(state["values"])
            out["info"] = ds.execute("refactorization")
    out["x"] = ds.execute("solve", None, b)
    if c["structure"] == "G":
        ds.setparam("solve_mode", 1)
        out["xt"] = ds.execute("solve", None, state["bt"])
        ds.setparam("solve_mode", 0)
    if c["family"] == "kkt":
        out["inertia"] = ds.getparam("inertia")
    return out


# -- what a pass cannot do without -------------------------------------------------------------------------------

def work(case):
    """Floating-point operations of the factorization (the sum over the panels' columns of the rows below, squared)
    and of the sweeps; bytes of the values, the factor and the vectors, each once."""
    c = case
    es = 4 if c["precision"] == "fp32" else 8
    # the systems of an uneven batch are analysed one by one: their forest is the same
    mats = _systems(c, 0) if c["family"] == "uneven" else [_matrix(c, 0)]
    S = [analyze_csr(A, c["structure"], reordering=c["reordering"], amalgamation=(c["maxwidth"], 0.25, 8)) for A in mats]
    n, nnz = sum(A.shape[0] for A in mats), sum(A.nnz for A in mats)
    stored, flops = float(sum(s.nnz_stored for s in S)), float(sum(s.flops for s in S))
    lu = c["structure"] == "G"
    sides = 2 if lu else 1
    k = c["members"] if c["family"] == "lap2d" else 1
    vectors = 16.0 * n * c["nrhs"]
    solves = 2 if c["op"] == "grad" or lu else 1
    solve_flops = solves * (2.0 * 2.0 * stored) * c["nrhs"] * (1 + c["ir_steps"] if c["ir_tol"] == 0 else 2)
    factor_bytes = sides * es * stored
    if c["op"] == "solve":
        return {"bytes": k * (factor_bytes + solves * vectors), "flops": k * solve_flops}
    grad = 8.0 * nnz if c["op"] == "grad" else 0.0
    return {"bytes": k * (8.0 * nnz + grad + factor_bytes + solves * vectors),
            "flops": k * (sides * flops + solve_flops)}


def tolerance(case):
    # Measured against the known solutions over some 60 cases of the ranges, times four and rounded up. FP64, and FP32
    # factors with two refinement steps: 1.4e-15 (2-norm) and 1.2e-14 (largest). One refinement step of an FP32 factor
    # leaves its contraction, 1.3e-13. A KKT system stops at a relative residual anywhere below 1e-12, which its
    # condition number then multiplies: 4.4e-13 seen, of a bound near 1e-11.
    if case["family"] == "kkt":
        return {"rel": 1e-11, "max": 1e-9}
    if case["precision"] == "fp32" and case["ir_steps"] < 2:
        return {"rel": 1e-12, "max": 1e-10}
    return {"rel": 2e-14, "max": 1e-12}


def exact(case, seed):
    c = case
    n = _uneven_size(c) if c["family"] == "uneven" else _size(c)
    X = _solution(c, seed, n)
    if c["op"] == "grad":
        # A-bar = -Y X^T on the pattern; a stored entry of a symmetric structure is read once, from its lower
        # triangle, and collects both terms
        Y = _solution(c, seed, n, 1)
        A = _matrix(c, seed)
        r = np.repeat(np.arange(n), np.diff(A.indptr))
        q = A.indices
        X2, Y2 = X.reshape(n, -1), Y.reshape(n, -1)
        abar = -(Y2[r] * X2[q]).sum(1)
        if c["structure"] != "G":
            both = abar - (Y2[q] * X2[r]).sum(1)
            abar = np.where(r == q, abar, np.where(r > q, both, 0.0))
        return {"x": X, "abar": abar, "bbar": Y}
    out = {"x": X, "info": None}
    if c["structure"] == "G":
        out["xt"] = _solution(c, seed, n, 1)
    if c["family"] == "kkt":
        out["inertia"] = (c["nx"] * c["ny"], c["nj"])
    return out
