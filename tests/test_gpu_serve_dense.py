"""Large batches of the fast search (more than two queries a resident warp:
k_serve's dense form) against the same queries in batches of 600 (a block per
query): equal ids, distances (bits), counts and expansions, on hierarchies and
on a random graph with wide lists."""
import numpy as np
import pytest

from nnm.datasets import gaussian_mixture_u8

pytestmark = pytest.mark.gpu

NQ = 9_000


def compare(ix, q, beams, **kw):
    big = ix.search(q, beams=beams, mode="fast", **kw)
    nc = ne = 0
    for b in range(0, len(q), 600):
        s = ix.search(q[b:b + 600], beams=beams[b:b + 600], mode="fast", **kw)
        assert np.array_equal(s["ids"], big["ids"][b:b + 600])
        assert np.array_equal(s["dists"].view(np.uint32), big["dists"][b:b + 600].view(np.uint32))
        nc, ne = nc + s["ncmps"], ne + s["expansions"]
    assert nc == big["ncmps"] and ne == big["expansions"]


@pytest.mark.parametrize("n,d,metric", [(3_001, 17, "l2"), (3_001, 200, "l1"), (200_003, 16, "l2"), (200_003, 16, "chi2")])
def test_dense(ctx, n, d, metric):
    x = gaussian_mixture_u8(n, d=d, seed=1) + np.float32(0.5)
    h = ctx.hmerge(x, 10, 10, seed=1, rng="fast", metric=metric)
    ix = ctx.index(x, h["layers"], seed=3, metric=metric)
    q = np.resize(gaussian_mixture_u8(1_500, d=d, seed=1), (NQ, d)) + np.float32(1)
    beams = np.random.default_rng(1).integers(5, 300, NQ).astype(np.uint32)
    for entry in ("default", "flat"):
        compare(ix, q, beams, out_k=5, entry=entry)
    ix.close()


@pytest.mark.parametrize("n", [5_000, 200_003])
def test_wide_lists(ctx, n):
    r = np.random.default_rng(2)
    x = gaussian_mixture_u8(n, d=12, seed=3)
    lens = r.choice([0, 3, 60, 150], n, p=[0.05, 0.15, 0.4, 0.4])
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    adj = r.integers(0, n, int(off[-1])).astype(np.uint32)
    ix = ctx.index(x, [(off, adj)], seed=1)
    q = gaussian_mixture_u8(NQ, d=12, seed=3) + np.float32(0.5)
    beams = r.choice([1, 8, 40, 90, 400], NQ).astype(np.uint32)
    for width in (1, 4):
        ix.set_width(width)
        compare(ix, q, beams, out_k=1, entry="flat")
    ix.close()
