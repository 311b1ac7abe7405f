"""The reference's random streams on the device (mt19937 draws of the initial
graphs and cross samples, std::rand() of the shuffles) at the edges of their
kernels' units -- 454 mt19937 words per pair of rounds, 496 std::rand()
outputs per warp -- and at the seeds' extremes: whole builds against the
oracle, bit for bit (integers and exact distances, so the tolerance is 0)."""
import numpy as np
import pytest

from nnm.datasets import gaussian_mixture_u8

pytestmark = pytest.mark.gpu

KEYS = ("ids", "dists", "flags", "trace")


@pytest.mark.parametrize("seed", [0, 1, 2**31, 2**32 - 1])
# kgraph draws n (k + 2) words: 36, 448, 456, 908 and 21,000 of them
@pytest.mark.parametrize("n,k", [(9, 2), (56, 6), (57, 6), (227, 2), (1500, 12)])
def test_kgraph_streams(ctx, oracle, n, k, seed):
    x = gaussian_mixture_u8(n, d=24, seed=n)
    got, exp = ctx.kgraph(x, k, seed=seed, exact_trace=True), oracle.kgraph(x, k, seed)
    assert all(np.array_equal(got[key], exp[key]) for key in KEYS) and got["ncmps"] == exp["ncmps"]


# phases of one call that shorten, repeat and extend the stream: the leaves',
# the cross samples', H-Merge's levels
@pytest.mark.parametrize("op,n", [("smerge", 97), ("smerge", 2500), ("jmerge", 1301), ("hmerge", 1100)])
def test_streams_across_phases(ctx, oracle, op, n):
    x = gaussian_mixture_u8(n, d=24, seed=n)
    a = (10, 8) if op == "hmerge" else (10,)
    got, exp = getattr(ctx, op)(x, *a, seed=5, exact_trace=True), getattr(oracle, op)(x, *a, 5)
    assert all(np.array_equal(got[key], exp[key]) for key in KEYS) and got["ncmps"] == exp["ncmps"]


# Reverse lists around the sizes where their sort changes hands: 32 (one
# entry a lane), 256 (a warp in shared memory, then a block in place) and past
# it.  Every row's nearest neighbours include row 0, so its reverse list is
# about n long; `hubs` such rows share them.
@pytest.mark.parametrize("n,hubs", [(30, 1), (36, 1), (40, 3), (255, 1), (262, 2), (300, 1), (700, 2), (4500, 1)])
def test_hub_reverse_lists(ctx, oracle, n, hubs):
    r = np.random.default_rng(n)
    x = np.zeros((n, 48), np.float32)
    for i in range(hubs, n):  # far from each other, near the hubs
        x[i, r.choice(48, 3, replace=False)] = r.integers(60, 90, 3)
    x[:hubs] = r.integers(0, 9, (hubs, 48))
    got, exp = ctx.kgraph(x, 6, seed=n, exact_trace=True), oracle.kgraph(x, 6, n)
    assert all(np.array_equal(got[key], exp[key]) for key in KEYS) and got["ncmps"] == exp["ncmps"]


# H-Merge carries a level's truncated reverse lists into the next: carried
# and new entries together cross the same sizes at this cap
def test_carried_reverse_lists(ctx, oracle):
    x = gaussian_mixture_u8(1700, d=16, n_centres=4, seed=8)
    x[:3] = x.mean(0).round()
    got, exp = ctx.hmerge(x, 16, 8, seed=4, exact_trace=True), oracle.hmerge(x, 16, 8, 4)
    assert all(np.array_equal(got[key], exp[key]) for key in KEYS) and got["ncmps"] == exp["ncmps"]
