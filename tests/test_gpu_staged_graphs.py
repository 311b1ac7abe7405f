"""Staged merges of graphs that the caller gives (nnm_merge_init_sgraph takes
any local ids, in any order) against the oracle's steps on the same graphs."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def oracle_graphs(path, x, k, pre, g1, g2, seed):
    """The oracle's S-Merge of two given sub-graphs: ids, distances, flags."""
    so = os.path.join(str(path), "graphs_smerge.so")
    subprocess.run(["gcc", "-O2", "-shared", "-fPIC", os.path.join(HERE, "cpp", "graphs_smerge.c"), "-o", so, "-lm"],
                   check=True)
    n, d = x.shape
    ids, dists, flags = np.zeros((n, k), np.uint32), np.zeros((n, k), np.float32), np.zeros((n, k), np.uint8)
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    assert ctypes.CDLL(so).nno_smerge_graphs(p(x), n, d, k, pre, p(g1), p(g2), seed, p(ids), p(dists), p(flags)) == 0
    return ids, dists, flags


def staged_graphs(ctx, x, k, pre, g1, g2, seed, join):
    m = ctx.merge_session(x, k, seed=seed, join=join)
    try:
        m.init_sgraph(0, g1, 0)
        m.init_sgraph(pre, g2, 1)
        m.initial_graph("smerge", pre)
        m.nndescent("smerge", pre)
        m.merge2one(len(x))
        return m.read()
    finally:
        m.close()


def check(ctx, path, x, k, pre, g1, g2, seed, join="fp32"):
    got = staged_graphs(ctx, x, k, pre, g1, g2, seed, join)
    ids, dists, flags = oracle_graphs(path, x, k, pre, g1, g2, seed)
    assert np.array_equal(got["ids"], ids) and np.array_equal(got["flags"], flags)
    assert np.array_equal(got["dists"].view(np.uint32), dists.view(np.uint32))


@pytest.mark.parametrize("n,k", [(300, 2), (701, 8), (1200, 31)])
def test_rows_in_any_order(ctx, tmp_path, n, k):
    """Random neighbours: neither the pools' halves nor the compensation lists
    are ascending when merge2one walks them."""
    r = np.random.default_rng(n)
    x = r.integers(0, 40, (n, 24)).astype(np.float32)
    pre = n // 2
    g = [np.array([r.choice(size, k, replace=False) for _ in range(size)], np.uint32) for size in (pre, n - pre)]
    check(ctx, tmp_path, x, k, pre, g[0], g[1], 3)


def hub_case(n, k, seed):
    """Rows far from each other and near row 0 (n / 2: row n / 2 of the second
    half); two rows in three list that hub twice, the others once."""
    r = np.random.default_rng(seed)
    x = np.zeros((n, 48), np.float32)
    for i in range(n):
        x[i, r.choice(48, 3, replace=False)] = r.integers(60, 90, 3)
    pre = n // 2
    for hub in (0, pre):
        x[hub] = r.integers(0, 9, 48)
    g = []
    for size in (pre, n - pre):
        a = np.zeros((size, k), np.uint32)
        for i in range(size):
            a[i] = 1 + r.choice(size - 1, k, replace=False)
            a[i][a[i] == i] = 0
            if i:
                a[i, 0] = 0
                if i % 3:
                    a[i, 1] = 0
        g.append(a)
    return x, pre, g[0], g[1]


@pytest.mark.parametrize("n,k", [(6000, 8), (20000, 6)])
def test_repeated_rows_across_sorted_runs(ctx, tmp_path, n, k):
    """Reverse lists of more than 4,096 entries that hold rows twice: the
    block-wide sort joins runs of 4,096 entries, and both copies of a row have
    to come through when they lie in different runs."""
    x, pre, g1, g2 = hub_case(n, k, n)
    check(ctx, tmp_path, x, k, pre, g1, g2, 7)
