"""The tensor-core join's tile loop where it can go wrong, against the FP32
join, bit for bit: operand rows of every chunk count of the gather (a row's
16-byte chunks over 2, 4 or 8 lanes, one to six 128-byte columns), fewer tiles
than CTAs or than producer groups, each form of the pair filter, and, for the
reduced-precision kinds, targets with few and with many exact sums in a flush
(dimensions around a stage's 16 floats)."""
import numpy as np
import pytest

from nnm.datasets import gaussian_mixture_u8

pytestmark = pytest.mark.gpu


def same(a, b):
    assert np.array_equal(a["ids"], b["ids"])
    assert np.array_equal(a["dists"].view(np.uint32), b["dists"].view(np.uint32))
    assert np.array_equal(a["flags"], b["flags"])
    assert a["ncmps"] == b["ncmps"] and a["iterations"] == b["iterations"]


def real_rows(n, d, seed):
    rng = np.random.default_rng(seed)
    c = rng.standard_normal((8, d)) * 3
    return (c[rng.integers(0, 8, n)] + rng.standard_normal((n, d))).astype(np.float32)


@pytest.mark.parametrize("rng", ["exact", "fast"])
@pytest.mark.parametrize("kern,d", [("u8", 3), ("u8", 33), ("u8", 65), ("u8", 129), ("u8", 300), ("u8", 768),
                                    ("tensor", 2), ("tensor", 15), ("tensor", 17), ("tensor", 63), ("tensor", 127),
                                    ("tensor", 192), ("fp8", 5), ("fp8", 33), ("fp8", 97), ("fp8", 256)])
def test_operand_widths(ctx, kern, d, rng):
    if kern == "u8":
        # narrow values: squared distances stay below 2^24 at d = 768
        x = np.floor(gaussian_mixture_u8(1500, d=d, seed=d) / 4).astype(np.float32)
    else:
        x = real_rows(1500, d, d)
    kw = dict(seed=4, rng=rng)
    same(ctx.kgraph(x, 12, join="tensor" if kern == "u8" else kern, **kw), ctx.kgraph(x, 12, join="fp32", **kw))


@pytest.mark.parametrize("n", [20, 33, 130, 300])
@pytest.mark.parametrize("kern", ["u8", "tensor", "fp8"])
def test_few_tiles_and_every_filter(ctx, kern, n):
    x = gaussian_mixture_u8(n, d=48, seed=n) if kern == "u8" else real_rows(n, 48, n)
    join = "tensor" if kern == "u8" else kern
    for rng in ("exact", "fast"):
        for fn in (ctx.kgraph, ctx.smerge, ctx.jmerge):
            same(fn(x, 8, seed=2, rng=rng, join=join), fn(x, 8, seed=2, rng=rng, join="fp32"))
    if n >= 300:
        same(ctx.hmerge(x, 8, 8, seed=3, join=join), ctx.hmerge(x, 8, 8, seed=3, join="fp32"))


@pytest.mark.parametrize("kern", ["tensor", "fp8"])
@pytest.mark.parametrize("d", [4, 61, 64, 68])
def test_exact_sums_of_close_rows(ctx, kern, d):
    """Rows so close that the bound leaves most proposals to the exact sums."""
    rng = np.random.default_rng(d)
    x = (rng.standard_normal((1, d)) * 4 + rng.standard_normal((4000, d)) * 0.02).astype(np.float32)
    for tier in ("exact", "fast"):
        same(ctx.merge_leaves(x, 20, [1000, 900, 1100, 1000], seed=6, rng=tier, join=kern),
             ctx.merge_leaves(x, 20, [1000, 900, 1100, 1000], seed=6, rng=tier, join="fp32"))
