"""The solve's level launches on a pattern whose leaf level has more than 600
blocks (40^3 Helmholtz, MetisND: 1,369 blocks at level 0), so the leaf
chains take every column of a pass in one CTA per block while the upper
levels split the columns into groups of four; the forward chain items pull
their own right-hand sides and the backward chain sums the split dots'
partials.  Per column the operations are those of a one-column solve, so a
many-column solve agrees with single-column solves to rounding; every
column's backward error is at the FP64 level (the oracle's solve of this
size is checked elsewhere, against the same kernels on smaller patterns).
A block's values are published as they are, so no result may have the bit
pattern that stands for "not there yet": right-hand sides with NaN and
infinities must neither stall a chain nor reach another column."""
import numpy as np
import pytest

from oracle.oracle import backward_error
from rslab_b200 import CscMatrix, LdltSymbolic, Ordering, SolverSettings, matgen

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def factor40():
    a = matgen.c2_matrix(40)
    st = SolverSettings(ordering=Ordering.METIS_ND)
    sym = LdltSymbolic.analyze_with(a, st)
    e = sym.export()
    blocks = np.bincount(np.asarray(e["sn_level"]), weights=(np.asarray(e["sn_ncol"]) + 63) // 64)
    assert blocks.max() >= 600 and blocks.min() < 600  # wide and narrow levels both present
    return a, sym.factor(a, st)


@pytest.mark.parametrize("nrhs", [5, 16, 20])
def test_many_columns_match_single_column_solves(factor40, nrhs):
    a, f = factor40
    b = matgen.uniform_rhs(a.n, nrhs, 11, complex_=True)
    x = f.solve_many(b, nrhs)
    assert backward_error(a, x, b) <= 1e-13
    for c in sorted({0, nrhs // 2, nrhs - 1}):
        xc = f.solve(np.ascontiguousarray(b[:, c]))
        assert np.max(np.abs(x[:, c] - xc)) <= 1e-13 * np.max(np.abs(xc))


@pytest.mark.parametrize("dtype", [np.float64, np.complex128, np.float32, np.complex64])
@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("kind", ["chain", "tree"])
def test_nan_and_infinite_right_hand_sides(kind, use_graph, dtype):
    st = SolverSettings(use_graph=use_graph)
    if kind == "chain":  # one dense supernode: a chain of five blocks
        rng, n = np.random.default_rng(1), 300
        c, r = np.triu_indices(n)
        a = CscMatrix.from_triplets(n, r, c, np.where(r == c, 4.0 * n, rng.standard_normal(r.size)).astype(dtype))
        st.ordering = Ordering.NATURAL
    else:
        a = matgen.c3_matrix(11).astype(dtype)
    f = LdltSymbolic.analyze_with(a, st).factor(a, st)
    real = np.zeros(1, dtype).real.dtype
    word = np.dtype("u%d" % real.itemsize)
    ones = np.full(1, np.iinfo(word).max, word).view(real)[0]  # the NaN with every bit set
    for nrhs in (1, 5, 17):
        b = matgen.uniform_rhs(a.n, nrhs, 3).reshape(a.n, nrhs).astype(dtype)
        clean = f.solve_many(b, nrhs).reshape(a.n, nrhs)
        assert np.all(np.isfinite(clean))
        at = nrhs // 2
        others = np.arange(nrhs) != at
        for bad in (ones, real.type(np.nan), real.type(np.inf), real.type(-np.inf)):
            for row in (0, a.n // 2, a.n - 1):
                bb = b.copy()
                (bb.imag if np.iscomplexobj(bb) else bb)[row, at] = bad
                x = f.solve_many(bb, nrhs).reshape(a.n, nrhs)
                assert not np.isfinite(x[row, at])
                assert np.array_equal(x[:, others], clean[:, others])
        assert np.array_equal(f.solve_many(b, nrhs).reshape(a.n, nrhs), clean)
