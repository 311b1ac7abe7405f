"""Device memory that a context keeps after a call that builds no graph, and
of H-Merge's layers: at most 256 MB of each, the rest is given back."""
import numpy as np
import pytest

import nnm
from nnm.datasets import gaussian_mixture_u8

pytestmark = pytest.mark.gpu
MB = 1 << 20


def used():
    import torch
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def calls(c, x, d):
    r = np.random.default_rng(1)
    ids = r.integers(0, len(x), (len(x), 10)).astype(np.uint32)
    trip = r.integers(0, len(x), (200, 3)).astype(np.uint32)
    return (lambda: c.graph_recall(x, ids, np.arange(200, dtype=np.uint32)),
            lambda: c.mlp_grad(nnm.mlp_init(d, seed=1), x, trip))


# n x d x 4 bytes: 340 MB, 290 MB with as much again of unpadded rows
@pytest.mark.parametrize("n,d", [(700_000, 128), (600_000, 125)])
def test_recall_and_gradients(n, d):
    c = nnm.Context(0)
    small = gaussian_mixture_u8(1_000, d=d, seed=1)
    for f in calls(c, small, d):
        f()
    start = used()
    for f in calls(c, np.resize(small, (n, d)), d):
        f()
        assert used() - start <= 32 * MB
    # what builds hold stays theirs
    g = c.kgraph(small, 10, seed=1)
    for f in calls(c, np.resize(small, (n, d)), d):
        f()
    assert np.array_equal(c.kgraph(small, 10, seed=1)["ids"], g["ids"])
    c.close()


def test_hierarchy_lists():
    c = nnm.Context(0)
    x = np.resize(gaussian_mixture_u8(20_000, d=16, seed=1), (300_000, 16)) + \
        np.random.default_rng(1).integers(0, 9, (300_000, 1)).astype(np.float32)
    a = c.hmerge(x, 8, 4, seed=1, rng="fast")
    start = used()
    c.hmerge(x, 8, 60, seed=1, rng="fast")
    assert used() - start <= 32 * MB
    b = c.hmerge(x, 8, 4, seed=1, rng="fast")
    assert all(np.array_equal(p, q) for l, m in zip(a["layers"], b["layers"]) for p, q in zip(l, m))
    c.close()
