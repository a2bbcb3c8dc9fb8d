"""The mesh contact's grid cells for every coordinate: the device's function
compiled for the CPU, and on the GPU a mesh scene that holds NaN."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_cell_is_in_the_grid(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ is absent")
    exe = str(tmp_path / "tt_cell")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", os.path.join(HERE, "tt_cell.cpp"), "-o", exe],
                   check=True)
    bad, n = (int(v) for v in subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split())
    assert n > 10000 and bad == 0


@pytest.mark.gpu
def test_mesh_with_nan_runs(gpu_lib):
    """A cube of a pile with NaN coordinates: it touches nothing, the others
    go on as if it were not there, and the run ends without an error."""
    from parmec_gb300.engine import GpuEngine
    from test_meshcontact import cube_pile
    out = []
    for row in (None, 0, 2):
        m = cube_pile()
        for p in (1, 11):                                # a cube of each layer
            m.P.position[0:3, p] += 0.5 if row is None else 0.0
            if row is not None:
                m.P.position[row, p] = np.nan
        eng = GpuEngine()
        m.dem(300e-5, 1e-5, interval=1e9, engine=eng)
        n = m.parnum
        if row is not None:
            assert np.isnan(m.P.position[row, [1, 11]]).all()
        keep = [p for p in range(n) if p not in (1, 11)]
        out.append(np.concatenate([m.P.position[0:3, keep], m.P.linear[:, keep], m.P.force[:, keep]]))
        eng.close()
    assert np.array_equal(out[0].view(np.int64), out[1].view(np.int64))
    assert np.array_equal(out[0].view(np.int64), out[2].view(np.int64))
