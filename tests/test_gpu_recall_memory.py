"""graph_recall where the host cannot hold the evaluated rows' lists: an error
of the call, not the end of the process."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHILD = """
import resource, sys
sys.path.insert(0, sys.argv[1])
import numpy as np, nnm
x = np.random.default_rng(1).integers(0, 255, (2000, 16)).astype(np.float32)
c = nnm.Context(0)
ids = c.kgraph(x, 16, seed=1)["ids"]
few = np.arange(100, dtype=np.uint32)
r = c.graph_recall(x, ids, few, atop=16)
rows = np.zeros(40_000_000, np.uint32)  # 160 MB; their lists: 2.7 GB
used = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (used + (1 << 30), resource.RLIM_INFINITY))
try:
    c.graph_recall(x, ids, rows, atop=16)
    print("no error")
except nnm.NnmError as e:
    print("error", e)
print("same" if c.graph_recall(x, ids, few, atop=16) == r else "other")
"""


@pytest.mark.gpu
def test_no_host_memory():
    r = subprocess.run([sys.executable, "-c", CHILD, os.path.join(ROOT, "nn-merge_b200")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    out = r.stdout.splitlines()
    assert out[0].startswith("error") and "memory" in out[0] and out[1] == "same", r.stdout
