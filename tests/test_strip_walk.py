"""The row-streaming kernels' copies and stores, walked on the host (tests/strip_walk.cpp):
every copy reads inside the domain, every cell is stored, and no asynchronous copy is
still in flight when a warp leaves its strip, whose shared memory the next block takes."""

from __future__ import annotations

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _cuda_include():
    for nvcc in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc"):
        if nvcc:
            inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
            if os.path.exists(os.path.join(inc, "cuda_runtime.h")):
                return inc
    return None


@pytest.mark.skipif(shutil.which("g++") is None or _cuda_include() is None, reason="needs g++ and the CUDA headers")
def test_strips_read_and_store_their_domain_and_leave_no_copy_in_flight(tmp_path):
    exe = tmp_path / "walk"
    subprocess.run(["g++", "-O1", "-w", "-std=c++17", "-I", _cuda_include(), "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "river-basin-sim_b200", "csrc"), os.path.join(ROOT, "tests", "strip_walk.cpp"),
                    "-o", str(exe)], check=True)  # fmt: skip
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout
