"""The arrays of the mesh-contact pair list where device memory runs out: the
session's own code (pg_ttbuffers.h) compiled for the CPU with an allocator
that fails at each of its calls in turn."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def cuda_include():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")


def test_failed_allocations_leave_no_freed_pointer(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ is absent")
    exe = str(tmp_path / "tt_buffers")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", cuda_include(), os.path.join(HERE, "tt_buffers.cpp"), "-o", exe],
                   check=True)
    bad, tried = (int(v) for v in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split())
    assert tried > 70                                    # 30 arrays and the copies, four times over
    assert bad == 0
