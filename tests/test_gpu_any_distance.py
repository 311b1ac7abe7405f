"""Distances that are not plain non-negative numbers: the chi-square distance
of components of both signs (negative where a sum of components is) is ordered
as the reference orders it, and NaN distances (rows with NaN) leave pools of
valid, distinct rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
KEYS = ("ids", "flags", "trace")


def signed(n, d, seed):
    return np.random.default_rng(seed).normal(20, 25, (n, d)).round(1).astype(np.float32)


@pytest.mark.parametrize("n,d,k", [(300, 5, 3), (900, 24, 10), (2500, 40, 20)])
@pytest.mark.parametrize("op", ["kgraph", "smerge", "jmerge", "hmerge"])
def test_signed_chi_square_is_the_reference(ctx, oracle, op, n, d, k):
    x = signed(n, d, n)
    a = (k, k) if op == "hmerge" else (k,)
    got = getattr(ctx, op)(x, *a, seed=5, metric="chi2", exact_trace=True)
    exp = getattr(oracle, op)(x, *a, 5, metric="chi2")
    assert (exp["dists"] < 0).any()
    assert all(np.array_equal(got[key], exp[key]) for key in KEYS) and got["ncmps"] == exp["ncmps"]
    assert np.array_equal(got["dists"].view(np.uint32), exp["dists"].view(np.uint32))


def well_formed(g, n):
    ids = np.sort(g["ids"].astype(np.int64), 1)
    assert (ids >= 0).all() and (ids < n).all()
    return ids


@pytest.mark.parametrize("op", ["kgraph", "smerge", "jmerge", "hmerge"])
def test_signed_chi_square_fast_tier(ctx, op):
    x = signed(1500, 30, 1)
    a = (12, 12) if op == "hmerge" else (12,)
    g = getattr(ctx, op)(x, *a, seed=5, metric="chi2", rng="fast")
    ids = well_formed(g, len(x))
    assert (np.diff(ids, axis=1) > 0).all() and (np.diff(g["dists"], axis=1) >= 0).all()
    assert (g["dists"] < 0).any()


@pytest.mark.parametrize("k", [6, 20])
@pytest.mark.parametrize("rng", ["exact", "fast"])
@pytest.mark.parametrize("op,metric", [("kgraph", "l2"), ("smerge", "l2"), ("jmerge", "l1"), ("hmerge", "l2"),
                                       ("kgraph", "chi2")])
def test_rows_with_nan(ctx, op, metric, rng, k):
    r = np.random.default_rng(k)
    x = r.uniform(0, 50, (1200, 20)).astype(np.float32)
    bad = r.choice(1200, 60, replace=False)
    x[bad, r.integers(0, 20, 60)] = np.nan
    x[bad[:5]] = np.inf
    a = (k, k) if op == "hmerge" else (k,)
    g = getattr(ctx, op)(x, *a, seed=5, metric=metric, rng=rng)
    well_formed(g, len(x))
    again = getattr(ctx, op)(x, *a, seed=5, metric=metric, rng=rng)
    assert np.array_equal(g["ids"], again["ids"])
    good = np.setdiff1d(np.arange(1200), bad)
    d = g["dists"][good]  # finite entries ascend, the others come last
    fin = np.isfinite(d)
    assert (np.diff(fin.astype(int), axis=1) <= 0).all()
    assert (np.diff(np.where(fin, d, np.float32(3e38)), axis=1) >= 0).all()
