"""The two forms of the exact search kernel on both sides of the lines between
them (descent: beam 48 + d while d < 128; flat: beam 48 + d/2, 256 at most) and
at a wide beam, with rows that tie, against the oracle bit for bit."""
import numpy as np
import pytest

from nnm.datasets import gaussian_mixture_u8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", ["l2", "l1", "chi2"])
@pytest.mark.parametrize("entry", ["default", "flat"])
@pytest.mark.parametrize("d", [4, 24, 61, 124, 128, 420])
def test_both_sides(ctx, oracle, d, entry, metric):
    n, nq, k = 3000, 9, 5
    x = np.floor(gaussian_mixture_u8(n, d=d, seed=d) / 32) + np.float32(0.5)
    x[::7] = x[3]  # equal rows: the heaps' order decides among them
    r = np.random.default_rng(d)
    up = np.arange(0, 201 * 6, 6).astype(np.uint64)[:201], r.integers(0, 200, 1200).astype(np.uint32)
    off = np.concatenate([[0], np.cumsum(r.integers(0, 45, n))]).astype(np.uint64)
    layers = [up, (off, r.integers(0, n, int(off[-1])).astype(np.uint32))]
    q = np.floor(gaussian_mixture_u8(nq, d=d, seed=d) / 32) + np.float32(1)
    dp = (d + 3) // 4 * 4
    line = min(48 + dp // 2, 256) if entry == "flat" else 48 + dp
    ix = ctx.index(x, layers, seed=11, metric=metric)
    try:
        for top in (line, line + 1, 900):
            beams = r.integers(k, top + 1, nq).astype(np.uint32)
            beams[0] = top
            exp = oracle.search_ex(x, layers, q, k, 11, beams=beams, flat=entry == "flat", metric=metric)
            got = ix.search(q, out_k=k, beams=beams, mode="exact", entry=entry)
            assert np.array_equal(got["ids"], exp["ids"]) and got["ncmps"] == exp["ncmps"]
            assert np.array_equal(got["dists"].view(np.uint32), exp["dists"].view(np.uint32))
    finally:
        ix.close()
