"""Panel kernels (k_getf2, k_deep) at the edges of their block widths, slot
columns and deep-row thresholds: a dense symmetric matrix in natural order is
one supernode, factored in blocks of panel_nb columns (128 from 512 columns).
With schur_engine="fma" every field must equal the oracle bit for bit (same
operations in the same order), pivots included."""
import numpy as np
import pytest

from oracle.oracle import OracleSolver
from rslab_b200 import CscMatrix, LdltSymbolic, Ordering, SolverSettings

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
                                  (513, 64), (600, 8)])
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
