"""Performance cases of the LDL^T path: what a program that uses rslab_b200 has it do, through its
public entry points, from a few hundred unknowns to the 64^3 Helmholtz factor.

A case is one call sequence of such a program:

  direct   new values on a factored pattern: `LdltSolver.refactor` + `solve_many` (host arrays)
  mixed    the refined pair: `MixedLdltSolver.refactor` + `solve_to(1e-14)` (page-locked host arrays)
  new      a factor handle per value set, as an interior-point or Newton loop makes it:
           `LdltSymbolic.factor` + `solve` (KKT systems: `solve_refined`, two corrections)
  solve    right-hand sides against a kept factor, in device memory: `LdltSolver.solve_device`
  sweep    frequencies of one pattern with static pivot reuse: `refactor` + `solve_to` for each
  batch    independent systems in one merged analysis: `MixedLdltSolver` in the FP64 tier
  gmres    block GMRES preconditioned by an incomplete factor: `krylov.gmres_block`

Matrices: 5- / 7-point Dirichlet Laplacians minus a shift (real: in a gap of the spectrum, so that the
condition number is that of the size and not an accident; complex: Helmholtz with 5% damping), scaled on
both sides by a seeded diagonal as a variable medium does; the 27-point sweep matrix K - w^2 M + i w C;
saddle-point (KKT) systems.  The grid matrices are diagonalised by sine transforms, which is how `exact`
solves them; the others are solved as dense matrices.
"""
from __future__ import annotations

import math
from functools import lru_cache

import numpy as np
import torch

from rslab_b200 import (CscMatrix, LdltSymbolic, MixedLdltSolver, Ordering, SolverSettings)
from rslab_b200 import _native as native
from rslab_b200 import batch as batching
from rslab_b200 import krylov

TARGET = 1e-14
NP = {"f64": np.float64, "c64": np.complex128, "f32": np.float32, "c32": np.complex64}
LOW = {"f32", "c32"}
UNIT = {"f64": 1.1e-16, "c64": 1.1e-16, "f32": 6.0e-8, "c32": 6.0e-8}


def _case(name, call, field, dims, nrhs, order="amd", method="left_looking", **more):
    c = {"name": name, "call": call, "matrix": "grid", "field": field, "dims": dims, "nrhs": nrhs, "order": order,
         "method": method}
    c.update(more)
    return c


def listed():
    return [
        # a control or circuit-sized grid: one new value set, one right-hand side; latency only
        _case("grid2d-tiny-f64", "direct", "f64", "24x20", 1),
        # an interior-point iteration: a fresh handle on a kept analysis, one solve
        _case("kkt-new-handle-f64", "new", "f64", "1400", 1, matrix="kkt"),
        # the 2D benchmark grid (128 x 128, real indefinite)
        _case("grid2d-128-f64", "direct", "f64", "128x128", 1),
        # time stepping: one right-hand side against a kept 3D factor
        _case("solve-1-f64", "solve", "f64", "37x40x33", 1),
        # many right-hand sides (sources, modes) against a kept complex factor: several passes
        _case("solve-40-c64", "solve", "c64", "33x30x35", 40, "metis"),
        # single precision asked for by the caller
        _case("grid3d-f32", "direct", "f32", "30x33x29", 3),
        # the multifrontal method on a real 3D grid
        _case("grid3d-multifrontal-f64", "direct", "f64", "31x34x30", 4, method="multifrontal"),
        # plain double precision on a complex 3D grid, nested dissection
        _case("helmholtz-fp64-c64", "direct", "c64", "44x41x43", 16, "metis"),
        # the refined pair on an uneven real 3D grid
        _case("grid3d-mixed-f64", "mixed", "f64", "36x29x41", 2),
        # a frequency sweep of the 27-point matrix, static pivots reused
        _case("sweep27-c64", "sweep", "c64", "24x24x24", 8, "metis", matrix="grid27", count=3),
        # a batch of uneven independent 3D systems, FP64 tier, every (system, column) certified
        _case("batch-f64", "batch", "f64", "12..24", 4, count=48),
        # the headline workload: 64^3 Helmholtz, single-precision factor refined to 1e-14, 16 right-hand sides
        _case("helmholtz-mixed-c64", "mixed", "c64", "64x64x64", 16, "metis"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    call = rng.choice(["direct", "direct", "mixed", "solve", "new", "sweep", "batch", "gmres"])
    nrhs = _log_int(rng, 1, 32)
    method = rng.choice(["left_looking", "left_looking", "multifrontal"])
    order = rng.choice(["amd", "metis"])
    if call == "new" and rng.random() < 0.5:
        return {"call": "new", "matrix": "kkt", "field": "f64", "dims": str(_log_int(rng, 200, 4000)), "nrhs": 1,
                "order": "amd", "method": "left_looking"}
    if call == "sweep":
        d = [rng.randint(6, 22) for _ in range(3)]
        return {"call": "sweep", "matrix": "grid27", "field": "c64", "dims": "x".join(map(str, d)), "nrhs": nrhs,
                "order": order, "method": "left_looking", "count": rng.randint(2, 4)}
    if call == "batch":
        lo = rng.randint(5, 12)
        return {"call": "batch", "matrix": "grid", "field": "f64", "dims": "%d..%d" % (lo, lo + rng.randint(1, 10)),
                "nrhs": min(nrhs, 8), "order": "amd", "method": "left_looking", "count": rng.randint(4, 64)}
    if rng.random() < 0.3:
        d = [_log_int(rng, 12, 180) for _ in range(2)]
    else:
        side = math.exp(rng.uniform(math.log(7), math.log(36)))
        d = [max(5, int(side * rng.uniform(0.8, 1.2))) for _ in range(3)]
    if call in ("mixed", "gmres"):
        field = rng.choice(["f64", "c64"])
    else:
        field = rng.choice(["f64", "c64", "f32", "c32"])
    if call == "gmres":
        nrhs, method = min(nrhs, 16), "left_looking"
    if call == "new":
        nrhs = 1
    return {"call": call, "matrix": "grid", "field": field, "dims": "x".join(map(str, d)), "nrhs": nrhs,
            "order": order, "method": method}


# ---------------------------------------------------------------------------
# Matrices.
# ---------------------------------------------------------------------------


def _dims(case):
    return [int(d) for d in case["dims"].split("x")]


def _eigs(dims):
    ev = np.zeros(1)
    for m in reversed(dims):  # the first dimension runs fastest
        ev = np.add.outer(ev, 2.0 - 2.0 * np.cos(np.arange(1, m + 1) * np.pi / (m + 1))).ravel()
    return ev


@lru_cache(maxsize=64)
def _shift(dims, field):
    """(shift, condition number of the shifted Laplacian).  Real fields: the middle of the widest gap of the
    spectrum near 0.1 lambda_max (2D: 0.3; single precision: 0.02, where the gaps are wider)."""
    ev = np.sort(_eigs(dims))
    top = ev[-1]
    if field in ("c64", "c32"):
        s = 0.2 * top * (1.0 + 0.05j)
    else:
        f = 0.02 if field in LOW else (0.3 if len(dims) == 2 else 0.1)
        ev = ev[np.concatenate([[True], np.diff(ev) > 1e-9])]  # the distinct eigenvalues
        near = ev[(ev >= 0.8 * f * top) & (ev <= 1.2 * f * top)]
        if near.size < 2:
            k = min(max(int(np.searchsorted(ev, f * top)), 1), ev.size - 1)
            near = ev[k - 1:k + 1]
        k = int(np.argmax(np.diff(near)))
        s = 0.5 * (near[k] + near[k + 1])
    a = np.abs(ev - s)
    return s, float(a.max() / a.min())


def _lower(dims, offsets):
    """Lower CSC pattern of a grid stencil: (col_ptr, row_idx, entry's column), the diagonal first in a column."""
    n = int(np.prod(dims))
    idx = np.arange(n)
    stride = np.cumprod([1] + list(dims[:-1]))
    pos = [(idx // stride[d]) % dims[d] for d in range(len(dims))]
    steps = sorted((int(np.dot(o, stride)), o) for o in offsets)
    rows = np.full((n, len(steps) + 1), -1, np.int64)
    rows[:, 0] = idx
    for k, (step, o) in enumerate(steps):
        ok = np.ones(n, bool)
        for d in range(len(dims)):
            ok &= (pos[d] + o[d] >= 0) & (pos[d] + o[d] < dims[d])
        rows[ok, k + 1] = idx[ok] + step
    keep = rows >= 0
    col_ptr = np.concatenate([[0], np.cumsum(keep.sum(axis=1))])
    return col_ptr, rows[keep], np.repeat(idx, keep.sum(axis=1))


def _grid(dims, field, seed):
    """(matrix, scaling d): diag(d) (Laplacian - shift) diag(d), rounded to the field; d depends on the seed."""
    offs = [tuple(int(i == d) for i in range(len(dims))) for d in range(len(dims))]
    cp, ri, cj = _lower(dims, offs)
    n = int(np.prod(dims))
    s, _ = _shift(tuple(dims), field)
    rng = np.random.default_rng(seed)
    # single precision: powers of two, so that the rounded matrix keeps its eigenvectors
    d = np.exp2(rng.integers(-1, 2, n)) if field in LOW else rng.uniform(0.7, 1.4, n)
    if field in LOW:
        s = complex(np.complex64(s)) if field == "c32" else float(np.float32(s))
    v = np.where(ri == cj, 2.0 * len(dims) - s, -1.0) * d[ri] * d[cj]
    return CscMatrix(n, cp, ri, v.astype(NP[field])), d


def _grid27(dims, seed, count):
    """The sweep matrices K - w^2 M + i w C at `count` frequencies of the band."""
    offs = [(x, y, z) for z in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1) if (z, y, x) > (0, 0, 0)]
    cp, ri, cj = _lower(dims, offs)
    n = int(np.prod(dims))
    rng = np.random.default_rng(seed)
    diag, mass = 26.0 + 0.1 * rng.random(n), 0.5 + rng.random(n)
    on = ri == cj
    k = np.full(len(ri), -1.0)
    k[on] = diag
    out = []
    for w in np.linspace(0.2, 1.1, count) * math.sqrt(26.05):
        v = k * (1.0 + 0.01j * w)
        v[on] -= w * w * mass
        out.append(CscMatrix(n, cp, ri, v))
    return out


def _kkt(nv, seed):
    """Saddle point [[H, J^T], [J, -1e-8 I]]: H diagonal plus a band, entries over four decades as an
    interior-point iteration has them; J nv / 3 rows of 4 entries."""
    rng = np.random.default_rng(seed)
    pat = np.random.default_rng(nv)  # the pattern belongs to the size, the values to the seed
    nc = nv // 3
    i = np.arange(nv)
    rows, cols, vals = [i], [i], [10.0 ** rng.uniform(-2, 2, nv) + 1.0]
    for o in (1, 7):
        rows.append(i[o:])
        cols.append(i[:-o])
        vals.append(rng.uniform(-0.4, 0.4, nv - o))
    jc = (np.arange(nc)[:, None] * 3 + np.array([0, 1, 2])[None, :]) % nv
    far = pat.integers(0, nv, nc)
    rows += [np.repeat(nv + np.arange(nc), 3), nv + np.arange(nc), nv + np.arange(nc)]
    cols += [jc.ravel(), far, nv + np.arange(nc)]
    vals += [rng.uniform(0.5, 1.5, 3 * nc), rng.uniform(0.1, 0.5, nc), np.full(nc, -1e-8)]
    return CscMatrix.from_triplets(nv + nc, np.concatenate(rows), np.concatenate(cols), np.concatenate(vals))


def _sides(case):
    lo, hi = (int(v) for v in case["dims"].split(".."))
    rng = np.random.default_rng(case["count"])
    return [int(v) for v in rng.integers(lo, hi + 1, case["count"])]


def _settings(case):
    s = SolverSettings()
    if case["call"] == "sweep":
        s = SolverSettings.preconditioner(1e-10)
    s.ordering = Ordering.METIS_ND if case["order"] == "metis" else Ordering.AMD
    s.method = case["method"]
    if case["call"] == "gmres":
        s.drop_tol = 1e-4
    return s


def _rhs(n, nrhs, field, seed):
    rng = np.random.default_rng(seed + 1_000_003)
    b = rng.uniform(-1, 1, (n, nrhs))
    if field in ("c64", "c32"):
        b = b + 1j * rng.uniform(-1, 1, (n, nrhs))
    b = b.astype(NP[field])
    return b[:, 0].copy() if nrhs == 1 else b


def _pinned(a):
    p = torch.empty(a.nbytes, dtype=torch.uint8, pin_memory=True).numpy().view(a.dtype).reshape(a.shape)
    p[...] = a
    return p


def _matrices(case, seed):
    if case["matrix"] == "kkt":
        return [_kkt(int(case["dims"]), seed)]
    if case["matrix"] == "grid27":
        return _grid27(_dims(case), seed, case["count"])
    if case["call"] == "batch":
        return [_grid([s] * 3, case["field"], seed * 1000 + k)[0] for k, s in enumerate(_sides(case))]
    return [_grid(_dims(case), case["field"], seed)[0]]


# ---------------------------------------------------------------------------
# What a program keeps, and one pass.
# ---------------------------------------------------------------------------


def prepare(case, seed):
    call, nrhs, field = case["call"], case["nrhs"], case["field"]
    mats = _matrices(case, seed)
    opts = _settings(case)
    st = {"call": call, "nrhs": nrhs, "opts": opts, "kkt": case["matrix"] == "kkt"}
    if call == "batch":
        systems = batching.BatchSystems(mats)
        sym = batching.analyze_batch(systems, opts)
        mats = [systems.as_matrix()]
        st["solver"] = MixedLdltSolver.factor_tier(mats[0], native.TIER_FP64, opts, sym=sym)
    else:
        sym = LdltSymbolic.analyze_with(mats[0], opts)
        if call in ("mixed", "sweep"):
            st["solver"] = MixedLdltSolver.factor_with(mats[0], opts, sym=sym)
        elif call != "new":
            st["solver"] = sym.factor(mats[0], opts)
    if call == "sweep":
        st["solver"].reuse_pivots(True)
    b = _rhs(mats[0].n, nrhs, field, seed)
    if call == "solve":
        st["b"] = torch.from_numpy(b).cuda()
        st["x"] = torch.empty_like(st["b"])
    else:
        for a in mats:
            a.values = _pinned(a.values)
        st["b"] = _pinned(b)
        st["out"] = [_pinned(np.empty_like(b)) for _ in mats]
    st.update(sym=sym, mats=mats)
    return st


def run(st):
    call, b, mats, solver = st["call"], st["b"], st["mats"], st.get("solver")
    if call == "direct":
        solver.refactor(mats[0])
        return solver.solve(b) if st["nrhs"] == 1 else solver.solve_many(b, st["nrhs"])
    if call == "new":
        f = st["sym"].factor(mats[0], st["opts"])
        return f.solve_refined(mats[0], b, 2) if st["kkt"] else f.solve(b)
    if call == "solve":
        solver.solve_device(b.data_ptr(), st["nrhs"], st["x"].data_ptr())
        return st["x"]
    if call == "gmres":
        solver.refactor(mats[0])
        r = krylov.gmres_block(solver, b, 1e-10)
        return r.x
    xs = []
    for a, out in zip(mats, st["out"]):
        solver.refactor(a)
        x, _ = solver.solve_to(a, b, TARGET, out=out)
        xs.append(x)
    return xs


@lru_cache(maxsize=64)
def _model(key):
    """(stored entries, factor entries, real flops of a factor and of a one-column solve, n) of a case."""
    case = dict(key)
    mats = _matrices(case, 1)
    nnz, n = sum(a.nnz for a in mats), sum(a.n for a in mats)
    if case["matrix"] == "grid27":
        mats = mats[:1]
    opts = _settings(case)
    fill = flops = 0.0
    for a in mats:
        i = LdltSymbolic.analyze_with(a, opts).info()
        fill += float(i.factor_nnz_sym)
        flops += float(i.flops_model)
    return nnz, n, fill, flops


def work(case):
    """One pass: values and right-hand sides in, solutions out, the multiply-adds of the factor and of one solve
    per right-hand side; for the solve calls the factor is an input, read once.  (Refinement steps beyond the
    first solve, and the Krylov steps, are not counted.)"""
    nnz, n, fill, flops = _model(tuple(sorted(case.items())))
    cx = case["field"] in ("c64", "c32")
    es = np.dtype(NP[case["field"]]).itemsize
    steps = case.get("count", 1) if case["call"] == "sweep" else 1
    nv = n // steps if case["call"] == "sweep" else n
    solve = 4.0 * fill * case["nrhs"]
    if case["call"] == "solve":
        return {"bytes": es * (fill + 2.0 * n * case["nrhs"]), "flops": solve * (4 if cx else 1)}
    return {"bytes": es * (nnz + (1.0 + steps) * nv * case["nrhs"]),
            "flops": steps * (flops + solve) * (4 if cx else 1)}


# ---------------------------------------------------------------------------
# 64-bit solutions and tolerances.
# ---------------------------------------------------------------------------


def _sine(m, dev):
    k = torch.arange(1, m + 1, dtype=torch.float64, device=dev)
    return torch.sin(k[:, None] * k[None, :] * (math.pi / (m + 1))) * math.sqrt(2.0 / (m + 1))


def _exact_grid(dims, field, seed, b):
    """x with diag(d) (L - s) diag(d) x = b, by sine transforms in 64 bits."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    _, d = _grid(dims, field, seed)
    s, _ = _shift(tuple(dims), field)
    if field in LOW:
        s = 2.0 * len(dims) - complex(np.asarray(2.0 * len(dims) - complex(np.complex64(s)), np.complex64))
        s = s if field == "c32" else s.real
    cx = field in ("c64", "c32")
    dt = torch.complex128 if cx else torch.float64
    y = torch.from_numpy(np.array(b).reshape(b.shape[0], -1)).to(dev, dt)
    dd = torch.from_numpy(d).to(dev)[:, None]
    shape = list(reversed(dims)) + [y.shape[1]]

    def transform(v):
        v = v.reshape(shape)
        for ax, m in enumerate(reversed(dims)):
            v = torch.movedim(torch.tensordot(_sine(m, dev).to(dt), v, dims=([1], [ax])), 0, ax)
        return v.reshape(y.shape)

    ev = torch.from_numpy(_eigs(dims)).to(dev)[:, None] - s
    x = transform(transform(y / dd) / ev) / dd
    return x.reshape(b.shape) if b.ndim > 1 else x[:, 0]


def _dense_solve(a, b):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n = a.n
    col = np.repeat(np.arange(n), np.diff(a.col_ptr))
    v = torch.from_numpy(np.array(a.values)).to(dev)
    m = torch.zeros(n, n, dtype=v.dtype, device=dev)
    r, c = torch.from_numpy(np.array(a.row_idx)).to(dev), torch.from_numpy(col).to(dev)
    m[r, c] = v
    m[c, r] = v
    return torch.linalg.solve(m, torch.from_numpy(np.array(b).reshape(n, -1)).to(dev)).reshape(b.shape)


def exact(case, seed):
    mats = _matrices(case, seed)
    n = sum(a.n for a in mats) if case["call"] == "batch" else mats[0].n
    b = _rhs(n, case["nrhs"], case["field"], seed)
    if case["matrix"] != "grid":
        xs = [_dense_solve(a, b) for a in mats]
        return xs if case["call"] == "sweep" else xs[0]
    if case["call"] == "batch":
        at, xs = 0, []
        for k, s in enumerate(_sides(case)):
            xs.append(_exact_grid([s] * 3, case["field"], seed * 1000 + k, b[at:at + s ** 3]))
            at += s ** 3
        return [torch.cat(xs)]
    x = _exact_grid(_dims(case), case["field"], seed, b)
    return [x] if case["call"] == "mixed" else x


def tolerance(case):
    """Forward errors grow with the condition number of the shifted Laplacian (known from its spectrum), times
    the unit roundoff of the field or the residual that the call asks for."""
    if case["matrix"] in ("kkt", "grid27"):  # refined to the working precision
        return {"rel": 1e-12, "max": 1e-10}
    if case["call"] == "batch":
        cond = max(_shift((s,) * 3, case["field"])[1] for s in set(_sides(case)))
    else:
        cond = _shift(tuple(_dims(case)), case["field"])[1]
    unit = 1e-10 if case["call"] == "gmres" else UNIT[case["field"]]
    refined = case["call"] in ("mixed", "batch", "gmres")
    rel = min(0.03, (4.0 if refined else 16.0) * cond * unit)
    return {"rel": rel, "max": min(0.9, 100.0 * rel)}
