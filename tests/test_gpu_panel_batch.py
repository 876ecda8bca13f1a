"""Dense trailing blocks of many value sets factored in panels whose rows and
columns are solved (and packed for the tensor cores) by a launch of their own,
at the edges of its 256-row blocks.

The matrices are completely filled and diagonally dominant by a factor of two,
so |L| |U| is below 3 |A| in norm and the factors lie within 6 n 2^-24 of the
FP64 ones, relative to the largest entry of their column.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lu(A):
    A = A.astype(np.float64)
    for k in range(A.shape[0] - 1):
        A[k + 1:, k] /= A[k, k]
        A[k + 1:, k + 1:] -= np.outer(A[k + 1:, k], A[k, k + 1:])
    return A


@pytest.mark.parametrize("tc", [0, 64], ids=["fma", "tensor_cores"])
@pytest.mark.parametrize("n", [65, 319, 320, 321, 577])
def test_panels_of_many_value_sets(n, tc):
    from pyglu import _capi

    eng, ptr = _capi.engine(), _capi.ptr
    sets = 592 // (1 + 2 * ((n - 64 + 127) // 128)) + 1
    rng = np.random.default_rng(n)
    v = rng.uniform(-1.0, 1.0, (sets, n, n)).astype(np.float32)  # [set][column][row]
    i = np.arange(n)
    v[:, i, i] = 0.0
    v[:, i, i] = 2.0 * np.maximum(np.abs(v).sum(1), np.abs(v).sum(2)) + 1.0
    check = [0, sets // 2, sets - 1]
    refs = [_lu(v[k].T) for k in check]
    ap = np.arange(n + 1, dtype=np.uint32) * n
    ai = np.tile(np.arange(n, dtype=np.uint32), n)
    sym, h = C.c_void_p(), C.c_void_p()
    _capi.check(eng.glu_symbolic_analyze(n, n * n, ptr(ap), ptr(ai), C.byref(sym)))
    _capi.check(eng.glu_create(sym, 0, sets, C.byref(h)))
    eng.glu_symbolic_destroy(sym)
    try:
        t = _capi.Tuning()
        _capi.check(eng.glu_get_tuning(h, C.byref(t)))
        t.dense_lookahead, t.dense_tc_min = 64, tc
        _capi.check(eng.glu_set_tuning(h, C.byref(t)))
        _capi.check(eng.glu_profile_enable(h, 1))
        _capi.check(eng.glu_load_lu_values(h, 0, sets, ptr(v), _capi.GLU_HOST, None))
        _capi.check(eng.glu_factor(h, 0, sets, 0, None))
        _capi.check(eng.glu_store_lu_values(h, 0, sets, ptr(v), _capi.GLU_HOST, None))
        assert _capi.kernel_times(h)["k_dense_panel"][1] > 0
    finally:
        eng.glu_destroy(h)
    for k, R in zip(check, refs):
        F = v[k].T.astype(np.float64)
        assert (np.abs(F - R).max(0) <= 6 * n * 2.0 ** -24 * np.abs(R).max(0)).all()
