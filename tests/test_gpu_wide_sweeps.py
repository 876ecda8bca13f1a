"""Solve sweeps over wide supernodes: with the inverses of their diagonal
blocks, and column by column where those could not be allocated; one and many
right-hand sides.

The matrices are block tridiagonal with filled blocks of the given width,
diagonally dominant by a factor of two (so the FP32 solution is within
18 n 2^-24 of the FP64 one, relative to the largest entry), in natural order
and without a dense trailing block.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(width, blocks, seed):
    rng = np.random.default_rng(seed)
    n = width * blocks
    at = np.arange(n) // width
    A = np.where(np.abs(at[:, None] - at[None, :]) <= 1, rng.uniform(-1.0, 1.0, (n, n)), 0.0)
    np.fill_diagonal(A, 0.0)
    np.fill_diagonal(A, 2.0 * np.maximum(np.abs(A).sum(0), np.abs(A).sum(1)) + 1.0)
    return A


@pytest.mark.parametrize("inverses", [True, False], ids=["inverses", "columns"])
@pytest.mark.parametrize("nrhs", [1, 3, 40])
@pytest.mark.parametrize("width", [16, 17, 33, 64, 100])
def test_sweeps_over_wide_supernodes(width, nrhs, inverses):
    from pyglu import _capi

    eng, ptr = _capi.engine(), _capi.ptr
    A = _matrix(width, 4, width)
    n = A.shape[0]
    cols, rows = np.nonzero(A.T)
    ap = np.zeros(n + 1, np.uint32)
    ap[1:] = np.cumsum(np.bincount(cols, minlength=n))
    ai = rows.astype(np.uint32)
    sym, h = C.c_void_p(), C.c_void_p()
    _capi.check(eng.glu_symbolic_analyze(n, ai.size, ptr(ap), ptr(ai), C.byref(sym)))
    _capi.check(eng.glu_create(sym, 0, 1, C.byref(h)))
    try:
        t = _capi.Tuning()
        _capi.check(eng.glu_get_tuning(h, C.byref(t)))
        t.dense_tail_min = 1 << 31
        _capi.check(eng.glu_set_tuning(h, C.byref(t)))
        st = _capi.Stats()
        _capi.check(eng.glu_get_stats(h, C.byref(st)))
        assert st.dense_tail == 0 and st.supernodes < n / 4
        val = np.empty(st.nnz_lu, np.float32)
        eng.glu_predict_lu(sym, ptr(np.ascontiguousarray(A.T[cols, rows])), ptr(val))
        _capi.check(eng.glu_load_lu_values(h, 0, 1, ptr(val), _capi.GLU_HOST, None))
        if not inverses:  # the factorization's only allocation without a dense block
            _capi.check(eng.glu_debug_inject(None, _capi.GLU_INJECT_ALLOC_FAILURES, 1))
        _capi.check(eng.glu_factor(h, 0, 1, 0, None))
        _capi.check(eng.glu_debug_inject(None, _capi.GLU_INJECT_ALLOC_FAILURES, 0))
        b = np.random.default_rng(nrhs).uniform(-1.0, 1.0, (nrhs, n)).astype(np.float32)
        ref = np.linalg.solve(A, b.astype(np.float64).T).T
        for _ in range(3):  # launched one by one, captured, and as a graph
            x = np.empty_like(b)
            _capi.check(eng.glu_solve(h, 0, nrhs, ptr(b), ptr(x), _capi.GLU_HOST, None))
            assert np.abs(x - ref).max() <= 18 * n * 2.0 ** -24 * np.abs(ref).max()
    finally:
        eng.glu_destroy(h)
        eng.glu_symbolic_destroy(sym)
