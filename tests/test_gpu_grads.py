"""The code network's gradients at the edges of their kernels' tiles: 16-value
tiles of the input dimension, chunks of 64 rows and 256-row bias strides (a
triplet is three rows), against the float64 oracle.

Tolerance: a gradient value is one chain of R rounded additions over terms
whose own errors come from sums of d + 1 and 257 products, so its error is
below (R + d + 300) 2^-24 of the terms' absolute sum; with R <= 600, d <= 256
and an absolute sum of up to seven times the largest gradient (the triplet
terms cancel in part) that is 5e-4 of the largest."""
import numpy as np
import pytest

import mlp_oracle as mo
from nnm import mlp_init
from nnm.datasets import gaussian_mixture_u8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 4, 15, 16, 17, 50, 128, 250, 256])
@pytest.mark.parametrize("ntrip", [1, 5, 21, 22, 43, 85, 86, 200])
def test_gradient_tiles(ctx, d, ntrip):
    r = np.random.default_rng(d * 1000 + ntrip)
    m = mlp_init(d, seed=3)
    m["b1"] = (r.standard_normal(256) * 0.1).astype(np.float32)
    x = gaussian_mixture_u8(300, d=d, seed=d)
    tr = r.integers(0, 300, (ntrip, 3)).astype(np.uint32)
    loss, g = ctx.mlp_grad(m, x, tr)
    oloss, og = mo.loss_and_grad(m, x, tr)
    assert abs(loss - oloss) <= 5e-4 * max(1.0, abs(oloss))
    for k in ("w1", "b1", "w2", "b2"):
        assert np.abs(g[k] - og[k]).max() <= 5e-4 * max(np.abs(og[k]).max(), 1e-6), k
