"""Wide supernodes' diagonal blocks whose inverse is not to be had in FP32, or
whose unknowns are infinite: the sweeps solve them by substitution.
"""
import numpy as np
import pytest

from engine_handle import blocks, handle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [1, 3])
@pytest.mark.parametrize("width", [17, 33, 64])
def test_blocks_whose_inverse_overflows(width, nrhs):
    """U = R U0 C, U0 dominant by a factor of two, R and C powers of two graded against each other: U, U0^-1 b and
    the solution are within FP32's range, entries of U^-1 reach 2^139.

    Substitution does not see the scales (they are exact), so C x lies within 18 n 2^-24 of U0^-1 R^-1 b.
    """
    A = blocks(width, 3, width)
    n = A.shape[0]
    at = np.arange(n) // width
    U0 = np.where(at[:, None] == at[None, :], np.triu(A), 0.0).astype(np.float32).astype(np.float64)
    grade = np.round(80 * (np.arange(n) % width) / (width - 1))
    r, c = 2.0 ** -grade, 2.0 ** (grade - 75)
    b0 = np.random.default_rng(nrhs).uniform(-1.0, 1.0, (nrhs, n)).astype(np.float32).astype(np.float64)
    ref = np.linalg.solve(U0, b0.T).T
    with handle(A, dense=False) as H:
        H.load(0, r[:, None] * U0 * c)
        H.capi.check(H.factor())
        x = H.solve(0, b0 * r) * c
        assert np.abs(x - ref).max() <= 18 * n * 2.0 ** -24 * np.abs(ref).max()


@pytest.mark.parametrize("value", [np.inf, -np.inf, 3e38])
@pytest.mark.parametrize("width", [20, 64])
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
