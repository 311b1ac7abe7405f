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
