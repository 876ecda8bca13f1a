"""The dense trailing block's triangular sweeps at the edges of their 64-row
blocks and of their groups of right-hand sides, plain and transposed, for one
value set and for several at once.

The matrices are completely filled, so the whole factor is the dense block;
the ordering is the identity.  Row and column diagonal dominance (off-diagonal
sums at half the diagonal) keeps |A^-1| |L| |U| below 6 in norm, so the FP32
solution is within 3 gamma_n * 6 = 18 n 2^-24 of the FP64 one, relative to the
largest entry.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(n, seed):
    rng = np.random.default_rng(seed)
    A = rng.uniform(-1.0, 1.0, (n, n))
    np.fill_diagonal(A, 0.0)
    d = 2.0 * np.maximum(np.abs(A).sum(0), np.abs(A).sum(1)) + 1.0
    return A + np.diag(d)


def _handle(mats):
    from pyglu import _capi

    eng, ptr = _capi.engine(), _capi.ptr
    n = mats[0].shape[0]
    ap = np.arange(n + 1, dtype=np.uint32) * n
    ai = np.tile(np.arange(n, dtype=np.uint32), n)
    sym, h = C.c_void_p(), C.c_void_p()
    _capi.check(eng.glu_symbolic_analyze(n, n * n, ptr(ap), ptr(ai), C.byref(sym)))
    _capi.check(eng.glu_create(sym, 0, len(mats), C.byref(h)))
    slot = np.empty(n * n, np.uint32)
    _capi.check(eng.glu_symbolic_slots(sym, ptr(slot)))
    eng.glu_symbolic_destroy(sym)
    _capi.check(eng.glu_set_source(h, n * n, ptr(ap), ptr(ai), ptr(slot), None))
    vals = np.stack([np.ascontiguousarray(A.T).reshape(-1) for A in mats])
    _capi.check(eng.glu_load_source_values(h, 0, len(mats), ptr(vals), _capi.GLU_HOST, None))
    _capi.check(eng.glu_factor(h, 0, len(mats), 0, None))
    return h


@pytest.mark.parametrize("nrhs", [1, 2, 4, 5, 33])
@pytest.mark.parametrize("n", [64, 65, 127, 128, 129, 200, 641])
def test_sweeps_of_the_dense_block(n, nrhs):
    from pyglu import _capi

    eng = _capi.engine()
    mats = [_matrix(n, 10 * n + k) for k in range(2)]
    h = _handle(mats)
    try:
        st = _capi.Stats()
        _capi.check(eng.glu_get_stats(h, C.byref(st)))
        assert st.dense_tail >= min(n, 64)
        b = np.random.default_rng(n + nrhs).uniform(-1.0, 1.0, (nrhs, n)).astype(np.float32)
        for inst, A in enumerate(mats):
            for fn, M in ((eng.glu_solve, A), (eng.glu_solve_transposed, A.T)):
                x = np.empty_like(b)
                _capi.check(fn(h, inst, nrhs, _capi.ptr(b), _capi.ptr(x), _capi.GLU_HOST, None))
                ref = np.linalg.solve(M, b.astype(np.float64).T).T
                assert np.abs(x - ref).max() <= 18 * n * 2.0 ** -24 * np.abs(ref).max()
    finally:
        eng.glu_destroy(h)


@pytest.mark.parametrize("transposed", [0, 1])
@pytest.mark.parametrize("n,nrhs", [(65, 1), (130, 3), (200, 6)])
def test_refined_solves_of_several_value_sets(n, nrhs, transposed):
    from pyglu import _capi

    eng = _capi.engine()
    mats = [_matrix(n, 7 * n + k) for k in range(3)]
    h = _handle(mats)
    try:
        b = np.random.default_rng(n).uniform(-1.0, 1.0, (3, nrhs, n))
        x = np.empty_like(b)
        rs = _capi.RefineStats()
        _capi.check(eng.glu_solve_refined(h, 0, 3, nrhs, _capi.ptr(b), _capi.ptr(x), 1e-12, 10, transposed,
                                          _capi.GLU_HOST, C.byref(rs), None))
        for k, A in enumerate(mats):
            M = A.T if transposed else A
            r = b[k] - x[k] @ M.T
            assert (np.linalg.norm(r, axis=1) <= 1e-12 * np.linalg.norm(b[k], axis=1)).all()
    finally:
        eng.glu_destroy(h)
