"""Block diagonal matrices: one level of supernodes without rows below them,
narrow and wide, for few and for many value sets, one and several right-hand
sides.

Blocks dominant by a factor of two: the factors lie within 6 w 2^-24 of the FP64
ones, relative to the largest entry of their column, solutions within 18 w 2^-24
of the FP64 ones, relative to the largest entry of their block.
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


@pytest.mark.parametrize("sets", [1, 5, 160])
@pytest.mark.parametrize("widths", [[2] * 60, [10] * 30, [16, 17] * 6, [40] * 8, [64, 3, 33, 5, 7] * 4, [9] * 80,
                                    [40] + [9] * 79 + [17]])
def test_factors_and_solutions(widths, sets):
    n = sum(widths)
    ends = np.cumsum(widths)
    check = sorted({0, sets // 2, sets - 1})
    mats = {}
    for z in check:
        A = np.zeros((n, n))
        for i, (w, e) in enumerate(zip(widths, ends)):
            A[e - w:e, e - w:e] = blocks(w, 1, 1000 * z + i)
        mats[z] = A
    b = np.random.default_rng(n).uniform(-1.0, 1.0, (3, n)).astype(np.float32)
    with handle(mats[0], sets, dense=False) as H:
        for z in range(sets):
            H.load(z, mats.get(z, mats[0]))
        H.capi.check(H.factor(0, sets))
        for z in check:
            F, X, Y = H.factors(z), H.solve(z, b[:1]), H.solve(z, b)
            for w, e in zip(widths, ends):
                at = slice(e - w, e)
                R = _lu(mats[z][at, at])
                assert (np.abs(F[at, at] - R).max(0) <= 6 * w * 2.0 ** -24 * np.abs(R).max(0)).all()
                ref = np.linalg.solve(mats[z][at, at], b[:, at].astype(np.float64).T).T
                for x, r in ((X, ref[:1]), (Y, ref)):
                    assert np.abs(x[:, at] - r).max() <= 18 * w * 2.0 ** -24 * np.abs(r).max()
