"""The first search of a process loads only the kernels it may run: a call of
one query, 2 ms in a fresh process, took 28 ms when all forms of the fast
search were one module."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = """
import sys, time
sys.path.insert(0, sys.argv[1])
import numpy as np, nnm
from nnm.datasets import gaussian_mixture_u8
x = gaussian_mixture_u8(2000, d=64, seed=1)
c = nnm.Context(0)
h = c.hmerge(x, 10, 10, seed=1, rng="fast")
ix = c.index(x, h["layers"], seed=1)
t = time.perf_counter()
ix.search(x[:1], out_k=5, beam=20)
print("ms", (time.perf_counter() - t) * 1e3)
"""


@pytest.mark.gpu
def test_first_search_of_a_process():
    env = {k: v for k, v in os.environ.items() if k != "CUDA_MODULE_LOADING"}
    best = 1e9
    for _ in range(3):  # the first process may page the library in
        r = subprocess.run([sys.executable, "-c", CHILD, os.path.join(ROOT, "nn-merge_b200")], env=env, check=True,
                           capture_output=True, text=True)
        best = min(best, float(r.stdout.split("ms")[-1]))
    assert best < 12.0
