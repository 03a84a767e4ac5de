"""A factor that fails in one panel block while other blocks of the level and
the side streams' kernels start: every CTA must take one decision (stop or go
on), the call reports the rank deficiency, and the handle stays usable."""
import ctypes as C
import re
from pathlib import Path

import numpy as np
import pytest

from rslab_b200 import CscMatrix, LdltSymbolic, Ordering, SolverSettings, matgen
from rslab_b200 import _native as N
from rslab_b200.solver import LdltSolver, NumericallyRankDeficient

DEVICE = Path(__file__).resolve().parents[1] / "rslab_b200" / "csrc" / "device"


def test_kernels_read_the_failure_word_as_a_cta():
    """No kernel returns on its own thread's read of the word: a warp that saw another value than its neighbours
    would leave them without the barriers, the tensor memory or the control words that it initialises."""
    for f in sorted(DEVICE.glob("*.cuh")):
        src = f.read_text()
        assert not re.search(r"if \((fa\.)?status\[0\][^;]*return", src), f.name
        for body in re.split(r"__global__", src)[1:]:
            if "factor_failed" in body:  # before anything that only part of the CTA does
                head = body[body.index("{"):body.index("factor_failed")]
                assert "threadIdx" not in head and "__shared__ __align__(16) unsigned char" not in head, f.name


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float64, np.complex128, np.float32, np.complex64])
@pytest.mark.parametrize("engine", ["fma", "tensor"])
def test_failed_factor_of_many_blocks_leaves_the_handle_usable(engine, dtype):
    # many small systems of several levels; one column of a later one is zero
    parts = [matgen.c1_matrix(s) for s in (9, 14, 11, 17) * 12] + [matgen.c3_matrix(9)]
    n = sum(p.n for p in parts)
    at = np.cumsum([0] + [p.n for p in parts])
    rows = np.concatenate([p.row_idx + o for p, o in zip(parts, at)])
    cols = np.concatenate([np.repeat(np.arange(p.n), np.diff(p.col_ptr)) + o for p, o in zip(parts, at)])
    vals = np.concatenate([p.values for p in parts]).astype(dtype)
    a = CscMatrix.from_triplets(n, rows, cols, vals)
    st = SolverSettings(schur_engine=engine)
    sym = LdltSymbolic.analyze_with(a, st)
    f = sym.factor(a, st)
    ref = f.export_factors()
    col = np.repeat(np.arange(n), np.diff(a.col_ptr))
    for system in (0, 20, len(parts) - 1):
        for rep in range(4):
            j = at[system] + 5 + 7 * rep
            bad = a.values.copy()
            bad[(col == j) | (a.row_idx == j)] = 0.0
            with pytest.raises(NumericallyRankDeficient):
                f.refactor(CscMatrix(n, a.col_ptr, a.row_idx, bad))
    f.refactor(a)
    g = f.export_factors()
    for k in ("two_by_two", "perm", "d_diag", "d_subdiag", "l_values"):
        assert np.array_equal(getattr(g, k), getattr(ref, k)), k


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float64, np.complex64])
def test_pivot_reuse_before_any_block_has_a_record(dtype):
    """Pivot reuse on a handle whose only factor failed in its first block: the steps without a record are taken in
    place, which on a dominant matrix is what the search chooses too."""
    n = 193
    rng = np.random.default_rng(1)
    c, r = np.triu_indices(n)
    v = rng.standard_normal(r.size).astype(dtype)
    v[r == c] += 4 * n
    a = CscMatrix.from_triplets(n, r, c, v)
    st = SolverSettings(ordering=Ordering.NATURAL, scaling="identity", schur_engine="fma")
    sym = LdltSymbolic.analyze_with(a, st)
    ref = sym.factor(a, st).export_factors()
    h, fs, zero = C.c_void_p(), st._factor_c(None), np.zeros_like(a.values)
    code = {np.float64: N.F64, np.complex64: N.C32}[dtype]
    assert N.lib.rslab_factor(sym._h, code, zero.ctypes.data_as(C.c_void_p), 0, C.byref(fs), C.byref(h)) != 0 and h
    f = LdltSolver(h, sym, dtype)
    f.reuse_pivots(True)
    f.refactor(a)
    g = f.export_factors()
    for k in ("two_by_two", "perm", "d_diag", "l_values"):
        assert np.array_equal(getattr(g, k), getattr(ref, k)), k
