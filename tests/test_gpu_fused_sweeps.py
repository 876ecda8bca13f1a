"""Supernodal sweeps as one launch each (sn_sweep_fused), over single columns,
narrow and wide supernodes, for several right-hand sides and value sets.

Diagonally dominant by a factor of two: FP32 solutions lie within 18 n 2^-24 of
the FP64 ones, relative to the largest entry.
"""
import numpy as np
import pytest

from engine_handle import blocks, handle

pytestmark = pytest.mark.gpu


def _tree(n, seed):
    """A random tree's matrix, parents behind their children: one column each."""
    rng = np.random.default_rng(seed)
    A = np.zeros((n, n))
    for i in range(n - 1):
        p = min(n - 1, i + 1 + int(rng.integers(0, 20)))
        A[i, p], A[p, i] = rng.uniform(-1.0, 1.0, 2)
    np.fill_diagonal(A, 2.0 * np.maximum(np.abs(A).sum(0), np.abs(A).sum(1)) + 1.0)
    return A


@pytest.mark.parametrize("sets", [1, 3])
@pytest.mark.parametrize("make", [lambda z: _tree(600, 1), lambda z: blocks(1, 300, z), lambda z: blocks(9, 30, z),
                                  lambda z: blocks(40, 6, z)], ids=["tree", "columns", "narrow", "wide"])
def test_fused_sweeps(make, sets):
    mats = [make(z) * (1.0 + 0.25 * z) for z in range(sets)]
    n = mats[0].shape[0]
    b = np.random.default_rng(n).uniform(-1.0, 1.0, (5, n)).astype(np.float32)
    with handle(mats[0], sets, dense=False) as H:
        H.tune(sn_sweep_fused=1)
        for z, A in enumerate(mats):
            H.load(z, A)
        H.capi.check(H.factor(0, sets))
        for z, A in enumerate(mats):
            ref = np.linalg.solve(A, b.astype(np.float64).T).T
            for nrhs in (1, 5):
                x = H.solve(z, b[:nrhs])
                assert np.abs(x - ref[:nrhs]).max() <= 18 * n * 2.0 ** -24 * np.abs(ref).max()
