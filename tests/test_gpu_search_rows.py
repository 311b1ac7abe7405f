"""The exact search kernel's staged rows and split candidate heap at their
edges: vectors of one to many 16-byte units (odd and even), lengths and beams
at which fewer rows or none are staged, more candidates than its shared-memory
head of 256 holds, lists longer than a chunk -- against the oracle, bit for
bit (the sums keep the reference's order)."""
import numpy as np
import pytest

from nnm.datasets import gaussian_mixture_u8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 4, 20, 36, 128, 130, 300, 900, 2100, 4000])
@pytest.mark.parametrize("topk", [1, 60, 700])
def test_dims(ctx, oracle, d, topk):
    x = gaussian_mixture_u8(1200, d=d, seed=d) + np.float32(0.5)
    h = ctx.hmerge(x, 12, 12, seed=1, rng="fast", join="fp32")
    q = gaussian_mixture_u8(6, d=d, seed=d) + np.float32(0.25)
    exp = oracle.search_ex(x, h["layers"], q, topk, 5, beams=np.full(6, topk, np.uint32))
    got = ctx.search(x, h["layers"], q, topk, seed=5)
    assert np.array_equal(got["ids"], exp["ids"]) and got["ncmps"] == exp["ncmps"]
    assert np.array_equal(got["dists"].view(np.uint32), exp["dists"].view(np.uint32))


@pytest.mark.parametrize("metric", ["l2", "l1", "chi2"])
def test_many_candidates(ctx, oracle, metric):
    """Wide lists and beams: thousands of candidates, ties among them."""
    r = np.random.default_rng(3)
    n = 5000
    x = np.floor(gaussian_mixture_u8(n, d=12, seed=4) / 16)
    lens = r.choice([0, 40, 97], n, p=[0.05, 0.55, 0.4])
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    adj = r.integers(0, n, int(off[-1])).astype(np.uint32)
    q = np.floor(gaussian_mixture_u8(20, d=12, seed=4) / 16) + np.float32(0.5)
    beams = r.integers(30, 1025, 20).astype(np.uint32)
    ix = ctx.index(x, [(off, adj)], seed=2, metric=metric)
    got = ix.search(q, out_k=30, beams=beams, mode="exact")
    ix.close()
    if metric == "l2":
        exp = oracle.search_ex(x, [(off, adj)], q, 30, 2, beams=beams)
        assert np.array_equal(got["ids"], exp["ids"]) and got["ncmps"] == exp["ncmps"]
        assert np.array_equal(got["dists"].view(np.uint32), exp["dists"].view(np.uint32))
    else:  # the oracle's extended search is L2: one query at a time gives the batch's results
        ix = ctx.index(x, [(off, adj)], seed=2, metric=metric)
        for i in range(20):
            one = ix.search(q[i:i + 1], out_k=30, beams=beams[i:i + 1], mode="exact")
            assert np.array_equal(one["ids"][0], got["ids"][i])
        ix.close()
