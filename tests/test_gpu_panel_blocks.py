"""Panel kernels (k_getf2, k_deep) at the edges of their block widths, slot
columns and deep-row thresholds: a dense symmetric matrix in natural order is
one supernode, factored in blocks of panel_nb columns (128 from 512 columns).
With schur_engine="fma" every field must equal the oracle bit for bit (same
operations in the same order), pivots included."""
import numpy as np
import pytest

from oracle.oracle import OracleSolver
from rslab_b200 import CscMatrix, LdltSymbolic, Ordering, SolverSettings
from rslab_b200.solver import ZeroPivotAction

pytestmark = pytest.mark.gpu


def dense_lower(n, dtype, dominant, seed):
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((n, n))
    if np.issubdtype(dtype, np.complexfloating):
        a = a + 1j * rng.standard_normal((n, n))
    a = a + a.T
    if dominant:
        a[np.arange(n), np.arange(n)] += 4.0 * n
    a[rng.random((n, n)) < 0.05] = 0.0  # exact zero multipliers
    c, r = np.triu_indices(n)  # column-major lower triangle
    return CscMatrix.from_triplets(n, r, c, a[r, c].astype(dtype))


@pytest.mark.parametrize("dtype", [np.float64, np.complex128, np.float32, np.complex64])
@pytest.mark.parametrize("n,nb", [(1, 64), (2, 64), (8, 64), (9, 64), (31, 64), (32, 64), (33, 64), (63, 64), (64, 64),
                                  (65, 64), (97, 64), (128, 64), (129, 64), (193, 64), (150, 17), (200, 128),
                                  (513, 64), (600, 8), (576, 64), (640, 64)])
def test_dense_panel_is_the_oracles(n, nb, dtype):
    for dominant in (False, True):
        a = dense_lower(n, dtype, dominant, n + nb)
        st = SolverSettings(ordering=Ordering.NATURAL, panel_nb=nb, schur_engine="fma")
        sym = LdltSymbolic.analyze_with(a, st)
        g = sym.factor(a, st).export_factors()
        o = OracleSolver(a, sym.export(), panel_nb=nb).factors()
        assert np.array_equal(g.two_by_two, o.two_by_two)
        assert np.array_equal(g.perm, o.perm)
        assert np.array_equal(g.d_diag, o.d_diag) and np.array_equal(g.d_subdiag, o.d_subdiag)
        assert np.array_equal(g.l_row_idx, o.l_row_idx) and np.array_equal(g.l_values, o.l_values)


def ldl_residual(a, f, cols=None):
    """Over columns [0, cols) of the lower triangles, in 64 bits and for identity scaling: the norms of
    P A P^T - L D L^T and of |L| |D| |L^T|."""
    n = a.n
    wide = np.complex128 if np.iscomplexobj(a.values) else np.float64
    L = np.eye(n, dtype=wide)
    below = f.l_row_idx > (col := np.repeat(np.arange(n), np.diff(f.l_col_ptr)))
    L[f.l_row_idx[below], col[below]] = f.l_values[below]
    D = np.diag(f.d_diag.astype(wide))
    for k in np.nonzero(f.two_by_two)[0]:
        D[k, k + 1] = D[k + 1, k] = f.d_subdiag[k]
    A = a.to_scipy_full().toarray().astype(wide)[np.ix_(f.perm, f.perm)]
    at = np.tril_indices(n, 0, n if cols is None else cols)
    return np.linalg.norm((A - L @ D @ L.T)[at]), np.linalg.norm((np.abs(L) @ np.abs(D) @ np.abs(L).T)[at])


@pytest.mark.parametrize("dtype", [np.float32, np.complex64, np.complex128])
@pytest.mark.parametrize("n,nb", [(1, 64), (31, 64), (32, 64), (33, 64), (63, 64), (64, 64), (65, 64), (128, 64), (129, 64),
                                  (193, 64), (150, 17), (200, 128), (513, 64), (600, 8), (640, 64)])
def test_fused_panels_at_their_edges(n, nb, dtype):
    """The tensor engine's instances (fused updates; pivots may differ from the oracle's): the factorization's
    backward error |P A P^T - L D L^T| against its bound n u |L| |D| |L^T|, with 2 sqrt(n) for n (rounding errors
    of random signs)."""
    for dominant in (False, True):
        a = dense_lower(n, dtype, dominant, n + nb)
        st = SolverSettings(ordering=Ordering.NATURAL, scaling="identity", panel_nb=nb, schur_engine="tensor")
        f = LdltSymbolic.analyze_with(a, st).factor(a, st).export_factors()
        assert np.array_equal(np.sort(f.perm), np.arange(n))
        r, s = ldl_residual(a, f)
        assert r <= 2.0 * np.sqrt(n) * np.finfo(dtype).eps / 2 * s


@pytest.mark.parametrize("dtype", [np.float64, np.complex128, np.float32, np.complex64])
@pytest.mark.parametrize("engine", ["fma", "tensor"])
@pytest.mark.parametrize("n,nb", [(33, 64), (65, 64), (193, 64), (200, 128), (640, 64)])
def test_replayed_interchanges_and_2x2_steps(n, nb, engine, dtype):
    a = dense_lower(n, dtype, False, n)
    st = SolverSettings(ordering=Ordering.NATURAL, panel_nb=nb, schur_engine=engine)
    f = LdltSymbolic.analyze_with(a, st).factor(a, st)
    g = f.export_factors()
    assert g.two_by_two.any() and not np.array_equal(g.perm, np.arange(n))
    f.reuse_pivots(True)
    f.refactor(a)
    h = f.export_factors()
    for k in ("two_by_two", "perm", "d_diag", "d_subdiag", "l_values"):
        assert np.array_equal(getattr(g, k), getattr(h, k)), k


@pytest.mark.parametrize("dtype", [np.float32, np.complex64, np.complex128])
@pytest.mark.parametrize("width,deep", [(33, 0), (64, 0), (128, 0), (64, 40), (64, 200)])
def test_fused_panel_rounds_no_more_than_the_reference(width, deep, dtype):
    """One block of a dominant matrix and its deep rows, fused (tensor engine) against the reference's operations: the
    fused form may not round an entry more often (10% for the luck of the draw; two roundings an update instead
    of one gave 1.3 to 2.2 times the residual)."""
    widths = (width, 30) if deep else (width,)
    n = sum(widths) + deep
    rng = np.random.default_rng(width + deep)
    full, at = np.zeros((n, n), np.complex128), 0
    for w in widths:
        full[at:, at:at + w] = rng.standard_normal((n - at, w)) + 1j * rng.standard_normal((n - at, w))
        full[at + w:n - deep, at:at + w] = 0.0  # the blocks are coupled through the last `deep` rows only
        at += w
    full[at:, at:] = rng.standard_normal((deep, deep))
    full = np.tril(full if np.issubdtype(dtype, np.complexfloating) else full.real)
    full[np.arange(n), np.arange(n)] += 4 * n
    r, c = np.nonzero(full)
    a = CscMatrix.from_triplets(n, r, c, full[r, c].astype(dtype))
    res = {}
    for engine in ("fma", "tensor"):
        st = SolverSettings(ordering=Ordering.NATURAL, scaling="identity", panel_nb=max(width, 64), schur_engine=engine)
        res[engine] = ldl_residual(a, LdltSymbolic.analyze_with(a, st).factor(a, st).export_factors(), width)[0]
    assert res["tensor"] <= 1.1 * res["fma"]


@pytest.mark.parametrize("dtype", [np.float64, np.complex128, np.float32, np.complex64])
@pytest.mark.parametrize("engine", ["fma", "tensor"])
def test_static_floor_above_1e19(dtype, engine):
    """Every third pivot (5e19) lies below the floor of 1e20; the others (5e21) and the updates (1e16) leave no doubt."""
    n = 40
    a = dense_lower(n, dtype, False, 3)
    v = a.values * dtype(1e18)
    v[a.row_idx == np.repeat(np.arange(n), np.diff(a.col_ptr))] = np.where(np.arange(n) % 3 == 0, 5e19, 5e21)
    a = CscMatrix(n, a.col_ptr, a.row_idx, v)
    st = SolverSettings(ordering=Ordering.NATURAL, scaling="identity", schur_engine=engine,
                        on_zero_pivot=ZeroPivotAction.perturb_to_eps(1e20))
    sym = LdltSymbolic.analyze_with(a, st)
    f = sym.factor(a, st)
    o = OracleSolver(a, sym.export(), perturb_floor=1e20, scaling=False).factors()
    assert f.n_perturbed() == o.n_perturbed == (n + 2) // 3
    g = f.export_factors()
    if engine == "fma":
        assert np.array_equal(g.d_diag, o.d_diag) and np.array_equal(g.l_values, o.l_values)
    else:  # at most 40 updates of a pivot, each rounded at its magnitude
        assert np.max(np.abs(g.d_diag - o.d_diag) / np.abs(o.d_diag)) <= 40 * np.finfo(dtype).eps


def test_wide_and_narrow_supernodes_of_one_level():
    """Blocks of 128, 64 and a few columns in the same launches, with few and
    many deep rows: leaves of one parent, in one matrix."""
    rng = np.random.default_rng(5)
    widths, sep = (600, 90, 40, 64, 5), 70
    n = sum(widths) + sep
    full = np.zeros((n, n))
    at = 0
    for w in widths:
        full[at:at + w, at:at + w] = rng.standard_normal((w, w))
        full[n - sep:, at:at + w] = rng.standard_normal((sep, w))
        at += w
    full[n - sep:, n - sep:] = rng.standard_normal((sep, sep))
    full = np.tril(full)
    r, c = np.nonzero(full)
    a = CscMatrix.from_triplets(n, r, c, full[r, c])
    for engine in ("fma", "tensor"):
        st = SolverSettings(ordering=Ordering.NATURAL, schur_engine=engine)
        sym = LdltSymbolic.analyze_with(a, st)
        g = sym.factor(a, st)
        o = OracleSolver(a, sym.export())
        b = rng.standard_normal(n)
        if engine == "fma":
            f, e = g.export_factors(), o.factors()
            assert np.array_equal(f.perm, e.perm) and np.array_equal(f.l_values, e.l_values)
        A = a.to_scipy_full()
        x, xo = g.solve(b), o.solve_many(b.reshape(n, 1), 1).reshape(n)
        scale = abs(A).sum(axis=1).max()
        be = [float(np.max(np.abs(b - A @ v)) / (scale * np.max(np.abs(v)) + np.max(np.abs(b)))) for v in (x, xo)]
        assert be[0] <= max(1e-13, 10 * be[1])
