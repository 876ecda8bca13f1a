"""Tensor-core updates under a wait limit too short for them: the call ends with
GLU_ERR_TIMEOUT or in time, and the same handle then factors correctly.

Filled matrices, dominant by a factor of two: the factors lie within
6 n 2^-24 of the FP64 ones, relative to the largest entry of their column.
"""
import numpy as np
import pytest

from engine_handle import blocks, handle

pytestmark = pytest.mark.gpu


def _lu(A):
    A = A.astype(np.float32).astype(np.float64)
    for k in range(A.shape[0] - 1):
        A[k + 1:, k] /= A[k, k]
        A[k + 1:, k + 1:] -= np.outer(A[k + 1:, k], A[k, k + 1:])
    return A


@pytest.mark.parametrize("lookahead", [0, 128])
def test_short_wait_limit_leaves_the_handle_usable(lookahead):
    sets = 2
    mats = [blocks(640, 1, z) for z in range(sets)]
    with handle(mats[0], sets) as H:
        H.tune(dense_lookahead=lookahead, dense_tc_min=64)
        H.capi.check(H.eng.glu_profile_enable(H.h, 1))
        for limit in (1, 0, 1, 0):
            H.capi.check(H.eng.glu_set_wait_limit(H.h, limit))
            for z, A in enumerate(mats):
                H.load(z, A)
            assert H.factor(0, sets) in ((H.capi.GLU_OK, H.capi.GLU_ERR_TIMEOUT) if limit else (H.capi.GLU_OK,))
            assert H.capi.kernel_times(H.h)["k_dense_update_tc"][1] > 0
        for z, A in enumerate(mats):
            R = _lu(A)
            assert (np.abs(H.factors(z) - R).max(0) <= 6 * H.n * 2.0 ** -24 * np.abs(R).max(0)).all()
