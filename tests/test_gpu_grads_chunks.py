"""The code network's gradients where k_grad_outer's chunks of 128 rows (three
to a triplet) end: just below one, whole chunks only (the prefetch stops on
the boundary), and one triplet more, against the float64 oracle.  Tolerance:
(R + d + 300) 2^-24 of the terms' absolute sum, at most seven times the largest
gradient, as derived for the smaller sizes; R = 387, d = 256: 4e-4 of the
largest."""
import numpy as np
import pytest

import mlp_oracle as mo
from nnm import mlp_init
from nnm.datasets import gaussian_mixture_u8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [3, 64, 256])
@pytest.mark.parametrize("ntrip", [42, 128, 129])
def test_gradient_chunks(ctx, d, ntrip):
    r = np.random.default_rng(d * 1000 + ntrip)
    m = mlp_init(d, seed=3)
    m["b1"] = (r.standard_normal(256) * 0.1).astype(np.float32)
    x = gaussian_mixture_u8(300, d=d, seed=d)
    tr = r.integers(0, 300, (ntrip, 3)).astype(np.uint32)
    loss, g = ctx.mlp_grad(m, x, tr)
    oloss, og = mo.loss_and_grad(m, x, tr)
    assert abs(loss - oloss) <= 4e-4 * max(1.0, abs(oloss))
    for k in ("w1", "b1", "w2", "b2"):
        assert np.abs(g[k] - og[k]).max() <= 4e-4 * max(np.abs(og[k]).max(), 1e-6), k
