"""Device memory that an index's searches keep: bounded whatever the batch,
and allocated for all batches once one has more blocks than the GPU has SMs."""
import numpy as np
import pytest

from nnm.datasets import gaussian_mixture_u8

pytestmark = pytest.mark.gpu
MB = 1 << 20


def used():
    import torch
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


# form: its batches, the first of which has more blocks (of four queries)
# than SMs; bound on what they keep, queries and results included: 4,144 warps
# of the fast form's bitmaps and lists of 16,384 ids
@pytest.mark.parametrize("mode,batches,most", [("fast", [3_100, 3_900, 5_000, 9_000, 20_000], 320),
                                               ("exact", [700, 900, 1_500, 2_400, 5_000], 1_000)])
def test_memory_of_growing_batches(ctx, mode, batches, most):
    x = gaussian_mixture_u8(50_000, d=16, seed=1)
    h = ctx.hmerge(x, 10, 10, seed=1, rng="fast")
    q = np.resize(gaussian_mixture_u8(2_000, d=16, seed=1), (batches[-1], 16)) + np.float32(1)
    ix = ctx.index(x, h["layers"], seed=3)
    start, after = used(), []
    for nq in batches:
        r = ix.search(q[:nq], out_k=10, beam=20, mode=mode)
        assert np.array_equal(r["ids"][:100], ix.search(q[:100], out_k=10, beam=20, mode=mode)["ids"])
        after.append(used() - start)
    assert after[-1] <= most * MB
    assert after[-1] - after[0] <= 24 * MB  # queries and results, not scratch
    ix.close()


@pytest.mark.parametrize("n", [33, 2_000, 40_000])
def test_more_visits_than_list_entries(ctx, n):
    """A warp per query, dense and not: queries that visit most of the layer
    (40,000 rows: more ids than a list holds) and few, in turn, give what a
    block per query gives."""
    r = np.random.default_rng(n)
    x = gaussian_mixture_u8(n, d=8, seed=2)
    deg = 24
    off = (np.arange(n + 1) * deg).astype(np.uint64)
    adj = r.integers(0, n, n * deg).astype(np.uint32)
    ix = ctx.index(x, [(off, adj)], seed=1)
    q = np.resize(gaussian_mixture_u8(300, d=8, seed=2), (9_000, 8)) + np.float32(0.5)
    beams = r.choice([1, 4, min(n, 1_000)], 9_000, p=[0.4, 0.4, 0.2]).astype(np.uint32)
    small = [ix.search(q[b:b + 300], beams=beams[b:b + 300], out_k=1, entry="flat") for b in range(0, 9_000, 300)]
    for nq in (4_500, 9_000):
        for _ in range(2):  # the second finds the bitmaps as the first left them
            big = ix.search(q[:nq], beams=beams[:nq], out_k=1, entry="flat")
            parts = small[:nq // 300]
            assert np.array_equal(big["ids"], np.concatenate([s["ids"] for s in parts]))
            assert big["ncmps"] == sum(s["ncmps"] for s in parts)
    ix.close()
