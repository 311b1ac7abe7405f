"""Queries and rows with NaN or infinity in the fast search, in its three
forms (a block per query; a warp per query; the dense one): a NaN distance
counts as infinite, so the beam holds distinct rows of the layer, the other
queries' results are what they are without such neighbours in the batch, and
a row with NaN is never before a finite one."""
import numpy as np
import pytest

from nnm.datasets import gaussian_mixture_u8

pytestmark = pytest.mark.gpu


def bad_queries(q):
    """Every 7th query: all NaN, one NaN, infinite, or an infinity that cancels
    against one of a row."""
    b = q.copy()
    at = np.arange(0, len(q), 7)
    b[at[0::4]] = np.nan
    b[at[1::4], 3] = np.nan
    b[at[2::4]] = np.inf
    b[at[3::4], 0] = np.inf
    return b, at


@pytest.mark.parametrize("nq", [200, 4_000, 9_000])
@pytest.mark.parametrize("metric,d", [("l2", 24), ("chi2", 24), ("l1", 140)])
def test_bad_queries_and_rows(ctx, nq, metric, d):
    x = gaussian_mixture_u8(3_001, d=d, seed=d) + np.float32(0.5)
    h = ctx.hmerge(x, 10, 10, seed=1, rng="fast", metric=metric)
    q = gaussian_mixture_u8(nq, d=d, seed=d) + np.float32(1)
    b, at = bad_queries(q)
    beams = np.random.default_rng(1).integers(10, 300, nq).astype(np.uint32)
    for rows in (x, x.copy()):
        if rows is not x:
            rows[5::50, 0] = np.inf
            rows[6::50, 1] = np.nan
        ix = ctx.index(rows, h["layers"], seed=3, metric=metric)
        for entry in ("default", "flat"):
            good = ix.search(q, out_k=10, beams=beams, entry=entry, mode="fast")
            got = ix.search(b, out_k=10, beams=beams, entry=entry, mode="fast")
            keep = np.setdiff1d(np.arange(nq), at)
            assert np.array_equal(got["ids"][keep], good["ids"][keep])
            assert np.array_equal(got["dists"][keep].view(np.uint32), good["dists"][keep].view(np.uint32))
            for r in (good, got):
                filled = np.sort(r["ids"], 1)
                assert (r["ids"] < len(x)).all() and (np.diff(filled.astype(np.int64), axis=1) > 0).all()
                dd = r["dists"].astype(np.float64)
                assert not np.isnan(dd).any() and (dd[:, 1:] >= dd[:, :-1]).all()
            assert np.isinf(got["dists"][at[0::4]]).all() and np.isinf(got["dists"][at[1::4]]).all()
        ix.close()
