"""Graphs of a handle's launch sequences: none is made for a sequence that few
calls make, and the calls that replay one see the values, value sets and
switches of their own.

Diagonally dominant by a factor of two: FP32 solutions lie within 18 n 2^-24 of
the FP64 ones, relative to the largest entry.
"""
import collections

import numpy as np
import pytest

from engine_handle import blocks, handle

pytestmark = pytest.mark.gpu


def _calls(f):
    """How often the runtime's functions were called in f."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    torch.zeros(1, device="cuda")
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        f()
    return collections.Counter(e.name for e in p.events())


def test_a_single_refined_solve_makes_no_graph():
    A = blocks(33, 4, 1)
    b = np.random.default_rng(2).uniform(-1.0, 1.0, A.shape[0])
    with handle(A, dense=False) as H:
        H.source([A])
        steps = []

        def use():
            H.capi.check(H.factor())
            steps.append(H.solve_refined(0, b, 0.0, 5)[1].iterations)

        calls = _calls(use)
        assert steps[0] >= 2  # the same sweeps three times and more
        assert calls["cudaLaunchKernel"] > 0 and calls["cudaStreamBeginCapture"] == 0, calls


def test_many_value_sets_in_turn_make_no_graph_after_graph():
    sets = 12  # more than a handle keeps graphs
    mats = [blocks(20, 4, k) for k in range(sets)]
    b = np.random.default_rng(2).uniform(-1.0, 1.0, mats[0].shape[0])
    with handle(mats[0], sets) as H:
        H.source(mats)

        def turn(rounds):
            for _ in range(rounds):
                H.source(mats)
                H.capi.check(H.factor(0, sets))
                for z in range(sets):
                    H.solve_refined(z, b, 0.0, 2)

        turn(10)
        calls = _calls(lambda: turn(3))
        # the factorization's graph outlives the solves' sequences
        assert calls["cudaStreamBeginCapture"] == 0 and calls["cudaGraphLaunch"] == 3, calls


@pytest.mark.parametrize("dense", [False, True], ids=["supernodes", "dense block"])
def test_replays_see_their_own_values(dense):
    sets, width = 3, 33
    keys = [(0, 3, 0), (0, 3, 1), (1, 2, 0), (2, 1, 1)]  # first, count, GESP
    b = np.random.default_rng(3).uniform(-1.0, 1.0, (2, 4 * width))
    n = b.shape[1]
    mats = [blocks(width, 4, k) for k in range(sets)]
    with handle(mats[0], sets, dense=dense) as H:
        for z in range(sets):
            H.load(z, mats[z])
        H.capi.check(H.factor(0, sets))
        for turn in range(12):
            for i, (first, count, perturb) in enumerate(keys):
                for z in range(first, first + count):
                    mats[z] = blocks(width, 4, 100 * turn + 10 * i + z)
                    H.load(z, mats[z])
                H.capi.check(H.factor(first, count, perturb))
                for z in range(sets):  # the others keep their factors
                    for nrhs in (1, 2):
                        ref = np.linalg.solve(mats[z], b[:nrhs].astype(np.float32).astype(np.float64).T).T
                        x = H.solve(z, b[:nrhs])
                        assert np.abs(x - ref).max() <= 18 * n * 2.0 ** -24 * np.abs(ref).max()
        assert _calls(lambda: H.solve(0, b))["cudaGraphLaunch"] == 1  # they were replays
