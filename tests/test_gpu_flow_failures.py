"""The waits of the dense block's dataflow factorization.

* A wait that runs out: no block takes the first tile
  (GLU_INJECT_UNSET_FACTOR_FLAG), so every wait for it gives up; the call
  returns GLU_ERR_TIMEOUT and the same handle then factors correctly.
* A wait limit far below the time that a tile waits in a sound factorization
  does not end one.

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


def _right(H, mats):
    for z, A in enumerate(mats):
        R = _lu(A)
        assert (np.abs(H.factors(z) - R).max(0) <= 6 * H.n * 2.0 ** -24 * np.abs(R).max(0)).all()


@pytest.mark.parametrize("sets", [1, 3])
@pytest.mark.parametrize("n", [80, 320, 577])
def test_wait_for_a_tile_runs_out_and_handle_stays_usable(n, sets):
    mats = [blocks(n, 1, n + z) for z in range(sets)]
    with handle(mats[0], sets) as H:
        capi, eng = H.capi, H.eng
        assert H.stats().dense_tail > 64
        for _ in range(3):
            for z, A in enumerate(mats):
                H.load(z, A)
            capi.check(eng.glu_set_wait_limit(H.h, 1000))
            capi.check(eng.glu_debug_inject(H.h, capi.GLU_INJECT_UNSET_FACTOR_FLAG, 0))
            assert H.factor(0, sets) == capi.GLU_ERR_TIMEOUT
            assert b"timed out" in eng.glu_last_error()
            capi.check(eng.glu_set_wait_limit(H.h, 0))
            for z, A in enumerate(mats):
                H.load(z, A)
            capi.check(H.factor(0, sets))
            _right(H, mats)


def test_a_short_limit_does_not_end_a_sound_factorization():
    mats = [blocks(577, 1, z) for z in range(4)]
    with handle(mats[0], 4) as H:
        H.capi.check(H.eng.glu_set_wait_limit(H.h, 1))
        for z, A in enumerate(mats):
            H.load(z, A)
        H.capi.check(H.factor(0, 4))
        _right(H, mats)


def test_unset_tile_injection_needs_a_dense_block():
    with handle(blocks(20, 4, 1), dense=False) as H:
        assert H.eng.glu_debug_inject(H.h, H.capi.GLU_INJECT_UNSET_FACTOR_FLAG, 0) == H.capi.GLU_ERR_UNSUPPORTED
