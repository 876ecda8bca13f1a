"""The dense trailing block factored by one dataflow launch (k_dense_flow), at
the edges of its 64 x 64 tiles, for one and for several value sets, with GESP
and at scales where the pivots leave the range of the quick quotient.

The matrices are completely filled, so the whole factor is the dense block,
and diagonally dominant by a factor of two, so |L| |U| is below 3 |A| in norm
and the factors lie within 2 * 3 gamma_n = 6 n 2^-24 of the FP64 ones, relative
to the largest entry of their column.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(n, seed, alone=()):
    """Dominant n x n matrix; the rows and columns in ``alone`` hold only a tiny diagonal."""
    rng = np.random.default_rng(seed)
    A = rng.uniform(-1.0, 1.0, (n, n))
    A[list(alone), :] = 0.0
    A[:, list(alone)] = 0.0
    np.fill_diagonal(A, 0.0)
    np.fill_diagonal(A, 2.0 * np.maximum(np.abs(A).sum(0), np.abs(A).sum(1)) + 1.0)
    for k in alone:
        A[k, k] = 1e-12
    return A


def _lu(A):
    A = A.astype(np.float32).astype(np.float64)
    for k in range(A.shape[0] - 1):
        A[k + 1:, k] /= A[k, k]
        A[k + 1:, k + 1:] -= np.outer(A[k + 1:, k], A[k, k + 1:])
    return A


def _factor(mats, perturb=0):
    """(factors as dense matrices, statistics): values in column order, dense pattern."""
    from pyglu import _capi

    eng, ptr = _capi.engine(), _capi.ptr
    n = mats[0].shape[0]
    ap = np.arange(n + 1, dtype=np.uint32) * n
    ai = np.tile(np.arange(n, dtype=np.uint32), n)
    sym, h = C.c_void_p(), C.c_void_p()
    _capi.check(eng.glu_symbolic_analyze(n, n * n, ptr(ap), ptr(ai), C.byref(sym)))
    _capi.check(eng.glu_create(sym, 0, len(mats), C.byref(h)))
    eng.glu_symbolic_destroy(sym)
    try:
        v = np.stack([np.ascontiguousarray(A.T, dtype=np.float32).reshape(-1) for A in mats])
        _capi.check(eng.glu_profile_enable(h, 1))
        _capi.check(eng.glu_load_lu_values(h, 0, len(mats), ptr(v), _capi.GLU_HOST, None))
        _capi.check(eng.glu_factor(h, 0, len(mats), perturb, None))
        _capi.check(eng.glu_store_lu_values(h, 0, len(mats), ptr(v), _capi.GLU_HOST, None))
        st = _capi.Stats()
        _capi.check(eng.glu_get_stats(h, C.byref(st)))
        kt = _capi.kernel_times(h)
        assert kt["k_dense_update"][1] == 1 and kt["k_dense_panel"][1] == 0, kt
        return [x.reshape(n, n).T.astype(np.float64) for x in v], st
    finally:
        eng.glu_destroy(h)


def _close(F, R, n):
    return (np.abs(F - R).max(0) <= 6 * n * 2.0 ** -24 * np.abs(R).max(0)).all()


@pytest.mark.parametrize("sets", [1, 3])
@pytest.mark.parametrize("n", [64, 65, 127, 128, 129, 200, 449])
def test_factors_of_filled_matrices(n, sets):
    mats = [_matrix(n, 5 * n + k) for k in range(sets)]
    for F, A in zip(_factor(mats)[0], mats):
        assert _close(F, _lu(A), n)


@pytest.mark.parametrize("scale", [1e-33, 1e33])
def test_pivots_outside_the_quick_quotients_range(scale):
    A = _matrix(130, 3) * scale
    assert _close(_factor([A])[0][0], _lu(A), 130)


@pytest.mark.parametrize("n", [65, 130])
def test_tiny_pivots_are_perturbed(n):
    """GESP replaces a tiny pivot of a column with an L part by +pert, and no other."""
    alone = sorted({0, 7, 63, n - 2, n - 1})
    A = _matrix(n, n, alone)
    (F,), st = _factor([A], perturb=1)
    R = _lu(A)
    for k in alone[:-1]:
        assert F[k, k] == st.pert
        F[k, k] = R[k, k]
    assert abs(F[n - 1, n - 1] - 1e-12) < 1e-18
    assert _close(F, R, n)
