"""Value sets factored one after another, the inverses of the wide supernodes'
diagonal blocks not to be had for the first of them: every set's solves use
inverses that were computed for it, or none.

Diagonally dominant by a factor of two, so the FP32 solution lies within
18 n 2^-24 of the FP64 one, relative to the largest entry.
"""
import numpy as np
import pytest

from engine_handle import blocks, handle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("failing", [0, 1], ids=["first factorization fails", "second factorization fails"])
def test_sets_factored_with_and_without_the_inverses(failing):
    from pyglu import _capi

    eng = _capi.engine()
    mats = [blocks(33, 4, k) for k in range(2)]
    n = mats[0].shape[0]
    b = np.random.default_rng(9).uniform(-1.0, 1.0, n)
    with handle(mats[0], sets=2, dense=False) as H:
        for z, A in enumerate(mats):
            H.load(z, A)
        for z in range(2):
            # without a dense block the inverses are a factorization's only allocation
            _capi.check(eng.glu_debug_inject(None, _capi.GLU_INJECT_ALLOC_FAILURES, int(z == failing)))
            try:
                _capi.check(H.factor(z))
            finally:
                _capi.check(eng.glu_debug_inject(None, _capi.GLU_INJECT_ALLOC_FAILURES, 0))
        for z, A in enumerate(mats):
            ref = np.linalg.solve(A, b.astype(np.float32).astype(np.float64))
            assert np.abs(H.solve(z, b) - ref).max() <= 18 * n * 2.0 ** -24 * np.abs(ref).max()
