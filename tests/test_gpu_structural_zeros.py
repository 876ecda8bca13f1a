"""Target columns of a supernode that lack its first rows: those structural
zeros take no part in the solve with the diagonal block, which need not be
finite there.
"""
import numpy as np
import pytest

from engine_handle import blocks, handle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("targets", [20, 100])
@pytest.mark.parametrize("width", [4, 8, 16, 17, 40, 64])
def test_columns_that_start_inside_the_supernode(width, targets, value):
    """Row z is the first that the columns behind the supernode have, so U(z, j) = A(z, j) whatever L(z, 0) is."""
    n, z = width + targets, width // 2
    A = blocks(n, 1, width)
    A[:z, width:] = 0.0
    with handle(A, dense=False) as H:
        H.load(0, A)
        H.capi.check(H.factor())
        assert (H.factors(0)[z, width:] == A[z, width:].astype(np.float32)).all()
        A[z, 0] = value
        H.load(0, A)
        assert H.factor() == H.capi.GLU_ERR_SINGULAR
        F = H.factors(0)
        assert not np.isfinite(F[z, z])
        assert (F[z, width:] == A[z, width:].astype(np.float32)).all()
