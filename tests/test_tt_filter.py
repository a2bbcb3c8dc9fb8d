"""The FP32 filter that chooses which distances of a triangle pair the mesh
contact takes in FP64, against the whole narrow phase: the device's own
functions compiled for the CPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_filter_keeps_every_deciding_distance(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ is absent")
    exe = str(tmp_path / "tt_filter")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(HERE, "tt_filter.cpp"),
                    "-o", exe], check=True)
    out = subprocess.run([exe, "400000"], check=True, capture_output=True, text=True).stdout.split()
    bad, apart, near, full = (int(v) for v in out[:4])
    assert bad == 0
    assert apart > 20000 and near > 20000 and full > 20000
