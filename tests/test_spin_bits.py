"""The short forms of the FP64 particle update (two-term exponential map,
settled gyroscopic term, unturned rotation) equal the general forms bit for
bit: the device's own functions compiled for the CPU, over random and special
values."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_short_forms_equal_general_forms(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ is absent")
    exe = str(tmp_path / "spin_bits")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(HERE, "spin_bits.cpp"),
                    "-o", exe], check=True)
    out = subprocess.run([exe, "1000000"], check=True, capture_output=True, text=True).stdout.split()
    cases, bad, spin, turn = (int(v) for v in out)
    assert cases == 6000000 and bad == 0
    assert spin > 100000 and turn > 100000
