"""bench.py --impl reference where the reference is not on the host: it says
so, and the oracle does not stand in for it."""
import argparse
import json
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


def absent(*a, **k):
    return None


def broken(*a, **k):
    raise RuntimeError("g++ failed:\n  details")


@pytest.mark.parametrize("build", [absent, broken])
def test_reference_arm_says_that_it_is_unavailable(build, monkeypatch, capsys):
    import bench
    from oracle import ispc_ref, pyoracle
    monkeypatch.setattr(ispc_ref, "build", build)

    def never(*a, **k):
        raise AssertionError("the oracle ran as the reference")
    monkeypatch.setattr(pyoracle, "OracleEngine", never)
    args = argparse.Namespace(spheres=2000, steps=1, warmup=3)
    assert bench.run_reference(args, 0, 1) == 0
    lines = capsys.readouterr().out.strip().splitlines()
    got = json.loads(lines[-1])
    assert got["impl"] == "reference" and "value" not in got
    assert got["unavailable"] and "\n" not in got["unavailable"]
    assert bench.run_reference(args, 1, 2) == 0
    assert not [l for l in capsys.readouterr().out.splitlines() if l.startswith("{")]
