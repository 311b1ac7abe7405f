"""H-Merge builds whose last level has fewer rows than its cross samples draw:
pools repeat ids, and the merge keeps the repeats as the reference does."""
import numpy as np
import pytest

from nnm.datasets import gaussian_mixture_u8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("join", ["auto", "fp32"])
@pytest.mark.parametrize("n", [65, 66, 70, 130, 258])
def test_small_last_level_is_the_reference(ctx, oracle, n, join):
    x = gaussian_mixture_u8(n, d=48, seed=n)
    got, exp = ctx.hmerge(x, 8, 8, seed=3, join=join), oracle.hmerge(x, 8, 8, 3)
    assert np.array_equal(got["ids"], exp["ids"]) and np.array_equal(got["flags"], exp["flags"])
    assert np.array_equal(got["dists"].view(np.uint32), exp["dists"].view(np.uint32))
    assert got["ncmps"] == exp["ncmps"]


@pytest.mark.parametrize("join", ["auto", "fp32"])
@pytest.mark.parametrize("levels,d", [(2, 8), (3, 6), (2, 20)])
def test_many_equal_distances_are_the_reference(ctx, oracle, levels, d, join):
    """Few distinct values: whole buffers of proposals at one distance, put in
    the reference's insert order after the sort by distance."""
    x = np.random.default_rng(d).integers(0, levels, (700, d)).astype(np.float32)
    for k, name in ((12, "kgraph"), (20, "smerge")):
        got, exp = getattr(ctx, name)(x, k, seed=5, join=join), getattr(oracle, name)(x, k, 5)
        assert np.array_equal(got["ids"], exp["ids"]) and np.array_equal(got["flags"], exp["flags"])
        assert np.array_equal(got["dists"], exp["dists"]) and got["ncmps"] == exp["ncmps"]
