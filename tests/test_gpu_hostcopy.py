"""Host copies through the pinned slots: builds from host arrays equal builds
from device memory at sizes around the thresholds (8 MB in, 8 MB out, chunk
remainders), from pageable and pinned memory, from several contexts at once,
and with a source that changes right after the call."""
import threading

import numpy as np
import pytest

import nnm
from nnm.datasets import gaussian_mixture_u8

pytestmark = pytest.mark.gpu


def dev_build(ctx, x, k, sizes):
    import torch
    t = torch.from_numpy(x).cuda()
    ids = torch.empty((len(x), k), dtype=torch.int32, device="cuda")
    ds = torch.empty((len(x), k), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    ctx.merge_leaves_dev(t.data_ptr(), x.shape[0], x.shape[1], k, sizes, ids.data_ptr(), ds.data_ptr(), seed=3, rng="fast")
    return ids.cpu().numpy().view(np.uint32), ds.cpu().numpy()


# x: n x d x 4 bytes; results: n x k x 9 bytes
@pytest.mark.parametrize("n,d,k", [(5000, 128, 10), (16383, 128, 10), (16384, 128, 10), (16385, 128, 10),
                                   (46603, 40, 20), (46604, 37, 20), (60133, 127, 31)])
@pytest.mark.parametrize("pinned", [False, True])
def test_sizes(ctx, n, d, k, pinned):
    import torch
    x = gaussian_mixture_u8(n, d=d, seed=n)
    if pinned:
        x = torch.from_numpy(x).pin_memory().numpy()
    sizes = [n // 2, n - n // 2]
    ids, ds = dev_build(ctx, x, k, sizes)
    g = ctx.merge_leaves(x, k, sizes, seed=3, rng="fast")
    assert np.array_equal(g["ids"], ids) and np.array_equal(g["dists"], ds)
    assert g["flags"].shape == (n, k) and g["flags"].max() <= 1


def test_index_and_results(ctx):
    """Vectors, lists and queries of several MB, results of 4 MB; the arrays
    are overwritten as soon as the call that took them returns."""
    x = gaussian_mixture_u8(60_001, d=64, seed=2)
    h = ctx.hmerge(x, 12, 12, seed=1, rng="fast")
    q = gaussian_mixture_u8(20_003, d=64, seed=2) + np.float32(1)
    xs, qs = x.copy(), q.copy()
    ix = ctx.index(xs, h["layers"], seed=1)
    xs[:] = 0
    r = ix.search(qs, out_k=25, beam=40)
    qs[:] = 0
    ref = np.concatenate([((q[i:i + 2000, None, :].astype(np.float64) - x[r["ids"][i:i + 2000].astype(np.int64)]) ** 2).sum(-1)
                          for i in range(0, len(q), 2000)])
    assert np.abs(ref - r["dists"]).max() <= 1e-5 * ref.max()
    ix.close()


def test_contexts_at_once():
    x = [gaussian_mixture_u8(20_000 + i, d=100, seed=i) for i in range(3)]
    alone, out = [], [None] * 3
    for v in x:
        c = nnm.Context(0)
        alone.append(c.kgraph(v, 16, seed=1)["ids"])
        c.close()

    def work(i):
        c = nnm.Context(0)
        for _ in range(3):
            out[i] = c.kgraph(x[i], 16, seed=1)["ids"]
        c.close()

    t = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    [v.start() for v in t]
    [v.join() for v in t]
    assert all(np.array_equal(a, b) for a, b in zip(alone, out))
