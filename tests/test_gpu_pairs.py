"""The FP32 join's staged pair kernels and their proposals at the list sizes
where tiers change hands (16, 32, 64, 128 entries), at vector lengths around
a shared-memory row, and where a tier's vectors no longer fit in shared
memory: whole builds against the oracle, bit for bit (the kernels keep the
reference's order of every float sum, so the tolerance is 0)."""
import numpy as np
import pytest

from nnm.datasets import vmf_mixture

pytestmark = pytest.mark.gpu

KEYS = ("ids", "dists", "flags", "trace")


def same(got, exp):
    return all(np.array_equal(got[key], exp[key]) for key in KEYS) and got["ncmps"] == exp["ncmps"]


# k and the sample cap set the list sizes: up to 2 (k + cap) entries
@pytest.mark.parametrize("metric", ["l2", "l1", "chi2"])
@pytest.mark.parametrize("d", [1, 4, 30, 33, 65])
@pytest.mark.parametrize("k", [3, 9, 24])
def test_tiers(ctx, oracle, metric, d, k):
    x = np.abs(vmf_mixture(700, d=d, n_centres=6, seed=d + k))
    assert same(ctx.kgraph(x, k, seed=7, metric=metric, exact_trace=True), oracle.kgraph(x, k, 7, metric=metric))


# tier 0 alone, all tiers but the last, none staged in shared memory
@pytest.mark.parametrize("d", [420, 900, 1800, 3700])
def test_long_vectors(ctx, oracle, d):
    x = vmf_mixture(160, d=d, n_centres=4, seed=d)
    assert same(ctx.jmerge(x, 12, seed=3, exact_trace=True), oracle.jmerge(x, 12, 3))


# zeros on both sides of a chi-square term, exact ties, the fast tier's form
def test_zeros_and_ties(ctx, oracle):
    x = np.floor(np.abs(vmf_mixture(900, d=20, n_centres=5, seed=2)) * 8) / 8
    assert same(ctx.smerge(x, 10, seed=1, metric="chi2", exact_trace=True), oracle.smerge(x, 10, 1, metric="chi2"))
    a, b = ctx.kgraph(x, 10, seed=1, rng="fast", join="fp32"), ctx.kgraph(x, 10, seed=1, rng="fast", join="fp32",
                                                                          graph=False)
    assert all(np.array_equal(a[key], b[key]) for key in ("ids", "dists", "flags"))
