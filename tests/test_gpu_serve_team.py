"""Small batches of the fast search (a block per query) against large ones (a
warp per query): the two keep the same beam and sum each distance in the same
tree, so ids, distances (bits), distance counts and expansions are equal.
Shapes at the edges: vectors of one, two and four float4 per lane, visited
bitmaps that end in a partial word, beams from 1 to 1,024, all entry modes and
step widths, lists longer than a chunk, empty lists and repeated ids."""
import numpy as np
import pytest

from nnm import entry_init
from nnm.datasets import gaussian_mixture_u8

pytestmark = pytest.mark.gpu

BIG = 4_500  # more queries than blocks of the per-query kernel are resident


def both(ix, q, **kw):
    """Results of the first len(q) of BIG queries, and of the same queries in
    a batch of their own."""
    n = len(q)
    beams = kw.pop("beams", None)
    fill = np.resize(np.arange(n), BIG)
    b = None if beams is None else beams[fill]
    big = ix.search(q[fill], beams=b, mode="fast", **kw)
    one = ix.search(q, beams=beams, mode="fast", **kw)
    assert np.array_equal(one["ids"], big["ids"][:n])
    assert np.array_equal(one["dists"].view(np.uint32), big["dists"][:n].view(np.uint32))
    if BIG % n == 0:  # the batch repeats the same queries: its counts are a multiple
        assert one["ncmps"] * (BIG // n) == big["ncmps"] and one["expansions"] * (BIG // n) == big["expansions"]


@pytest.mark.parametrize("d", [1, 30, 128, 132, 260, 512])
@pytest.mark.parametrize("metric", ["l2", "l1", "chi2"])
def test_dims_and_metrics(ctx, d, metric):
    x = gaussian_mixture_u8(3001, d=d, seed=d) + np.float32(0.25)
    h = ctx.hmerge(x, 10, 10, seed=2, rng="fast", metric=metric)
    ix = ctx.index(x, h["layers"], seed=4, metric=metric)
    q = gaussian_mixture_u8(9, d=d, seed=d) + np.float32(0.5)
    for entry, beam in (("default", 10), ("flat", 33), ("default", 200)):
        both(ix, q, out_k=10, beam=beam, entry=entry)
    both(ix, q[:1], out_k=1, beam=1, entry="default")
    ix.close()


def test_beams_widths_entries(ctx):
    x = gaussian_mixture_u8(20_011, d=100, seed=3)
    h = ctx.hmerge(x, 20, 20, seed=2, rng="fast")
    ix = ctx.index(x, h["layers"], seed=4)
    m = entry_init(100, ix.entry_layer()[1], seed=1)
    ix.entry_train(m, steps=40, seed=2)
    ix.set_entry_model(m, probes=5)
    q = gaussian_mixture_u8(90, d=100, seed=3) + np.float32(3)
    beams = np.random.default_rng(1).integers(1, 1025, 90).astype(np.uint32)
    for width in (1, 2, 3, 4):
        ix.set_width(width)
        for entry in ("default", "flat", "learned"):
            both(ix, q, out_k=1, beams=beams, entry=entry)
    ix.close()


def test_odd_lists(ctx):
    """One layer with empty lists, lists of 200 ids and repeated ids."""
    r = np.random.default_rng(6)
    n = 2_500
    x = gaussian_mixture_u8(n, d=20, seed=9)
    lens = r.choice([0, 1, 31, 32, 33, 64, 200], n, p=[0.1, 0.1, 0.2, 0.2, 0.2, 0.1, 0.1])
    lens[:50] = 200
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    adj = r.integers(0, n, int(off[-1])).astype(np.uint32)
    adj[::5] = adj[1::5][: len(adj[::5])] if len(adj[1::5]) >= len(adj[::5]) else adj[::5]
    ix = ctx.index(x, [(off, adj)], seed=1)
    q = gaussian_mixture_u8(10, d=20, seed=9) + np.float32(1)
    for entry in ("default", "flat"):
        for beam in (5, 64, 300, 1000):
            both(ix, q, out_k=5, beam=beam, entry=entry)
    ix.close()
