"""Column-by-column solve sweeps (no supernodes): columns and rows that end
inside, at and just past a work item, levels as launches of their own and as
runs inside one cluster, plain and transposed.

An arrow of the given reach (every column and row of the first block holds
that many entries) over a random sparse part, diagonally dominant by a factor
of two (so the FP32 solution is within 18 n 2^-24 of the FP64 one, relative to
the largest entry), in natural order and without a dense trailing block.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(reach, seed):
    rng = np.random.default_rng(seed)
    n = reach + 40
    keep = rng.random((n, n)) < 2.0 / n
    keep[:3, :reach + 1] = keep[:reach + 1, :3] = True
    A = np.where(keep, rng.uniform(-1.0, 1.0, (n, n)), 0.0)
    np.fill_diagonal(A, 0.0)
    np.fill_diagonal(A, 2.0 * np.maximum(np.abs(A).sum(0), np.abs(A).sum(1)) + 1.0)
    return A


@pytest.mark.parametrize("thin", [1, 1 << 20], ids=["levels", "cluster"])
@pytest.mark.parametrize("nrhs", [1, 3])
@pytest.mark.parametrize("reach", [3, 33, 127, 128, 129, 257])
def test_column_sweeps(reach, nrhs, thin):
    from pyglu import _capi

    eng, ptr = _capi.engine(), _capi.ptr
    A = _matrix(reach, reach)
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
        t.dense_tail_min, t.sn_width, t.solve_thin = 1 << 31, 0, thin
        _capi.check(eng.glu_set_tuning(h, C.byref(t)))
        st = _capi.Stats()
        _capi.check(eng.glu_get_stats(h, C.byref(st)))
        assert st.dense_tail == 0
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
