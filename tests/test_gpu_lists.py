"""Candidate lists of spheres at their limits, on the GPU: by eight lanes a
sphere (up to 32 entries) and by one thread a sphere (more)."""
import numpy as np
import pytest

from helpers import assert_bitwise, assert_spheres_bitwise, bits, make_collision_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kn", [32, 33])
def test_nan_spheres_fill_no_list(kn, gpu_lib):
    """48 spheres with a NaN coordinate, all in the border cells: they are
    nobody's partner, so no list runs out of room and the others go on as if
    they were not there."""
    from parmec_gb300.engine import GpuEngine
    out = []
    for z in (7.0, np.nan):
        m, dt = make_collision_scene(n_side=4, seed=4)
        first = m.parnum
        m.spheres(np.array([(0.15, 0.15, 5.0 + 0.05 * k) for k in range(48)]), np.full(48, 0.015), 0, 1)
        m.P.position[2, first:m.parnum] += z - 7.0
        eng = GpuEngine(capacity=(kn, 32))
        m.dem(30 * dt - 0.5 * dt, dt, interval=1e9, engine=eng)
        assert np.isnan(m.P.position[2, first:m.parnum]).all() == np.isnan(z)
        out.append([getattr(m.P, name)[..., :first] for name in ("position", "linear", "angular", "rotation", "force")])
        eng.close()
    for a, b in zip(*out):
        assert np.array_equal(bits(a), bits(b))
