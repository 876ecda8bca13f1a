"""Values at the end of FP32's range in factors and solves: an infinite
quotient stays infinite.
"""
import numpy as np
import pytest

from engine_handle import blocks, handle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.inf, -np.inf, 3e38])
@pytest.mark.parametrize("width", [1, 2, 8])
def test_infinite_unknown(width, value):
    """The last unknown of the U sweep is infinite (its right-hand side, or the quotient by a pivot below one)."""
    A = blocks(width, 2, width)
    A *= 2.0 ** -20
    n = A.shape[0]
    b = np.zeros(n)
    b[n - 1] = value
    with handle(A, dense=False) as H:
        H.load(0, A)
        H.capi.check(H.factor())
        assert H.solve(0, b)[n - 1] == np.sign(value) * np.inf


@pytest.mark.parametrize("dense", [False, True], ids=["supernode", "dense block"])
@pytest.mark.parametrize("row", [5, 20, 39])
def test_infinite_quotient_in_the_factors(row, dense):
    """L(row, 0) = 3e38 / 0.25 is infinite; the rest of column 0 are the quotients."""
    A = blocks(40, 1, row)
    A[0, 0] = 0.25
    A[row, 0] = 3e38
    with handle(A, dense=dense) as H:
        H.load(0, A)
        assert H.factor() == H.capi.GLU_ERR_SINGULAR  # the pivot of that row is not finite
        F = H.factors(0)
        assert F[row, 0] == np.inf
        rest = [i for i in range(1, 40) if i != row]
        assert (F[rest, 0] == (A[rest, 0].astype(np.float32) / np.float32(0.25))).all()
