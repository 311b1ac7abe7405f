"""The dense form of the fast search where its rule starts for wider beams
(L2 and L1, by the index's size: 64, 72 and 100 queries an SM): on both sides
of each line the results of a block per query, bit for bit."""
import numpy as np
import pytest

from nnm.datasets import gaussian_mixture_u8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric,n,d,beam,line", [("l2", 3_001, 20, 300, 64), ("l1", 60_000, 20, 100, 72),
                                                  ("l2", 60_000, 20, 300, 100), ("l1", 150_000, 8, 100, 100),
                                                  ("l2", 150_000, 132, 300, 100)])
def test_lines(ctx, metric, n, d, beam, line):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    x = gaussian_mixture_u8(n, d=d, seed=1) + np.float32(0.5)
    h = ctx.hmerge(x, 10, 10, seed=1, rng="fast", metric=metric)
    ix = ctx.index(x, h["layers"], seed=3, metric=metric)
    q = np.resize(gaussian_mixture_u8(600, d=d, seed=1) + np.float32(1), (line * sms + 1, d))
    exp = ix.search(q[:600], out_k=5, beam=beam)
    for nq in (line * sms, line * sms + 1):
        got = ix.search(q[:nq], out_k=5, beam=beam)
        at = np.arange(nq) % 600
        assert np.array_equal(got["ids"], exp["ids"][at])
        assert np.array_equal(got["dists"].view(np.uint32), exp["dists"][at].view(np.uint32))
    ix.close()
