"""Host copies (hostcopy.cu) on the CPU, over a stand-in for the CUDA runtime
whose copies run late and whose calls can fail (tests/cpp/hostcopy_main.cpp)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME") or (os.path.dirname(os.path.dirname(os.path.realpath(shutil.which("nvcc"))))
                                       if shutil.which("nvcc") else "/usr/local/cuda")


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")),
                    reason="needs g++ and the CUDA headers")
def test_copies_over_a_stand_in_runtime(tmp_path):
    exe = str(tmp_path / "hostcopy")
    subprocess.run(["g++", "-O1", "-g", "-std=c++17", "-pthread", "-I", os.path.join(CUDA, "include"),
                    os.path.join(ROOT, "tests", "cpp", "hostcopy_main.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-1000:]
