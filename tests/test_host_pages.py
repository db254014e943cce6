"""ready_pages (host_pages.h) on plain host memory, with a stand-in for CUDA's pointer query: a buffer in use
costs no query, a fresh one is asked about once, contents are kept; and no exception leaves it when there is
no memory for a helper thread."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "laboetie_gb300", "csrc")


@pytest.mark.skipif(not shutil.which("g++"), reason="no host compiler")
def test_queries_and_helpers(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    exe = str(tmp_path / "check")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-I", cuda,
                           os.path.join(HERE, "c_abi", "host_pages_check.cpp"), "-o", exe])
    lines = subprocess.check_output([exe], text=True).split("\n")[:-1]
    assert lines[:6] == [f"{b} {used} asked {1 - used} kept 1" for b in (1000, 300 << 10, 64 << 20) for used in (0, 1)]
    assert lines[6:] == [f"helpers {n}" for n in range(3)]
