"""The split point on patterns without fill to speak of: the dense trailing
block must not take columns whose work it multiplies.
"""
import numpy as np
import pytest

from engine_handle import handle

pytestmark = pytest.mark.gpu


def _blocks(width, count, border):
    """Filled diagonal blocks, and a border of filled rows and columns behind them."""
    n = width * count + border
    A = np.zeros((n, n))
    A[:width * count, :width * count] = np.kron(np.eye(count), np.ones((width, width)))
    A[width * count:, :] = 1.0
    A[:, width * count:] = 1.0
    np.fill_diagonal(A, 2.0 * n)
    return A


@pytest.mark.parametrize("sets", [1, 16])
@pytest.mark.parametrize("width,count,border", [(300, 20, 0), (32, 60, 100), (40, 50, 0), (1, 2000, 60)])
def test_dense_block_is_not_mostly_padding(width, count, border, sets):
    with handle(_blocks(width, count, border), sets) as H:
        st = H.stats()
        assert 2.0 / 3.0 * st.dense_tail ** 3 <= 4.0 * st.factor_flops, st.dense_tail
