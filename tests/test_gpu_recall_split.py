"""Recall with the data set split over blocks: row counts around the 64-row
tiles, the 16 rows of a block and the smallest shares, few and many evaluated
rows, against exact distances in 64-bit integers (integer data: every FP32
sum is exact, so the recall is exact)."""
import numpy as np
import pytest

from nnm.datasets import gaussian_mixture_u8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nrows,atop,d", [(2, 2, 1, 8), (17, 17, 16, 3), (63, 1, 10, 128), (64, 15, 10, 20),
                                            (65, 16, 16, 20), (513, 17, 1, 128), (1025, 33, 10, 36),
                                            (20001, 7, 10, 100), (5000, 2500, 16, 12), (700, 5, 10, 512)])
def test_recall_shares(ctx, n, nrows, atop, d):
    r = np.random.default_rng(n + d)
    x = gaussian_mixture_u8(n, d=d, seed=n)
    rows = r.choice(n, nrows, replace=False).astype(np.uint32)
    ids = r.integers(0, n, (n, 16)).astype(np.uint32)
    xi = x.astype(np.int64)
    hits = 0
    for i in rows:
        dd = ((xi - xi[i]) ** 2).sum(1)
        others = np.sort(np.delete(dd, i))
        near = np.argsort(dd, kind="stable")
        ids[i, ::2] = near[near != i][:8] if n > 8 else ids[i, ::2]
        kth = others[atop - 1] if atop <= n - 1 else np.inf
        hits += sum(1 for j in ids[i, :atop] if j != i and dd[j] <= kth)
    assert ctx.graph_recall(x, ids, rows, atop=atop) == hits / (nrows * atop)
