"""Coupling of the dense trailing block with the sparse unknowns in plain and
transposed solves: tail columns with equal and with differing rows, of lengths
at the edges of a lane's share, and counts of right-hand sides at those of a
block's.

The leading part is diagonal, the tail filled; the matrices are diagonally
dominant by a factor of two (so the FP32 solution is within 18 n 2^-24 of the
FP64 one, relative to the largest entry), in natural order.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(t, m, seed):
    rng = np.random.default_rng(seed)
    n = t + m
    keep = np.zeros((n, n), bool)
    keep[t:, t:] = True
    for j in range(m):  # neighbours alike in the first half, each its own in the second
        rows = np.arange(t) if j < m // 2 else rng.permutation(t)[:rng.integers(0, t + 1)]
        keep[rows, t + j] = True
        keep[t + j, rows] = True
    A = np.where(keep, rng.uniform(-1.0, 1.0, (n, n)), 0.0)
    np.fill_diagonal(A, 0.0)
    np.fill_diagonal(A, 2.0 * np.maximum(np.abs(A).sum(0), np.abs(A).sum(1)) + 1.0)
    return A


@pytest.mark.parametrize("nrhs", [1, 4, 5])
@pytest.mark.parametrize("m", [64, 71])
@pytest.mark.parametrize("t", [1, 63, 64, 65, 150])
def test_tail_coupling(t, m, nrhs):
    from pyglu import _capi

    eng, ptr = _capi.engine(), _capi.ptr
    A = _matrix(t, m, 100 * t + m)
    n = t + m
    cols, rows = np.nonzero(A.T)
    ap = np.zeros(n + 1, np.uint32)
    ap[1:] = np.cumsum(np.bincount(cols, minlength=n))
    ai = rows.astype(np.uint32)
    sym, h = C.c_void_p(), C.c_void_p()
    _capi.check(eng.glu_symbolic_analyze(n, ai.size, ptr(ap), ptr(ai), C.byref(sym)))
    _capi.check(eng.glu_create(sym, 0, 1, C.byref(h)))
    try:
        tu = _capi.Tuning()
        _capi.check(eng.glu_get_tuning(h, C.byref(tu)))
        tu.dense_tail_min = 32
        _capi.check(eng.glu_set_tuning(h, C.byref(tu)))
        st = _capi.Stats()
        _capi.check(eng.glu_get_stats(h, C.byref(st)))
        assert st.dense_tail >= 64
        val = np.empty(st.nnz_lu, np.float32)
        eng.glu_predict_lu(sym, ptr(np.ascontiguousarray(A.T[cols, rows])), ptr(val))
        _capi.check(eng.glu_load_lu_values(h, 0, 1, ptr(val), _capi.GLU_HOST, None))
        _capi.check(eng.glu_factor(h, 0, 1, 0, None))
        b = np.random.default_rng(nrhs).uniform(-1.0, 1.0, (nrhs, n)).astype(np.float32)
        for solve, M in ((eng.glu_solve, A), (eng.glu_solve_transposed, A.T)):
            ref = np.linalg.solve(M, b.astype(np.float64).T).T
            for _ in range(3):  # launched one by one, captured, and as a graph
                x = np.empty_like(b)
                _capi.check(solve(h, 0, nrhs, ptr(b), ptr(x), _capi.GLU_HOST, None))
                assert np.abs(x - ref).max() <= 18 * n * 2.0 ** -24 * np.abs(ref).max()
    finally:
        eng.glu_destroy(h)
        eng.glu_symbolic_destroy(sym)
