"""Spheres whose rotation is not finite, without a torque, in both particle
updates: NaN where the oracle has NaN, the others' bits equal."""
import numpy as np
import pytest

from helpers import STATE

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [20, 19457])
def test_rotation_that_is_not_finite(n, gpu_lib, oracle_lib):
    from oracle.pyoracle import OracleEngine
    from parmec_gb300.engine import GpuEngine
    from parmec_gb300.model import Model
    out = []
    for eng in (GpuEngine(), OracleEngine()):
        m = Model()
        mat = m.material(2500.0, 1e9, 0.25)
        side = 28
        g = np.stack(np.meshgrid(*(np.arange(side),) * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
        m.spheres(0.05 * g, np.full(n, 0.01), mat, 1)
        m.granular(0, 0, 1e6, 0.2, 0.5)
        m.set_gravity(0.0, 0.0, -9.81)
        for k, (entry, value, spin) in enumerate([(0, np.nan, 0.0), (4, np.nan, 5.0), (7, np.inf, 0.0), (2, -np.inf, 3.0),
                                                  (8, np.nan, -0.0), (None, 0.0, 2.0), (None, 0.0, 0.0)]):
            if entry is not None:
                m.P.rotation[entry, k] = value
            m.P.angular[0:3, k] = m.P.angular[3:6, k] = (0.0, spin, 0.5 * spin)   # finite, in both frames
        m.dem(4e-5, 1e-5, interval=1e9, engine=eng)
        out.append(m)
    a, b = out
    assert np.isnan(b.P.angular[0:3, :5]).any()
    for name in STATE:
        x, y = getattr(a.P, name)[..., :n], getattr(b.P, name)[..., :n]
        assert np.array_equal(np.isnan(x), np.isnan(y)), name
        ok = ~np.isnan(x)
        assert np.array_equal(x[ok].view(np.int64), y[ok].view(np.int64)), name
