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
