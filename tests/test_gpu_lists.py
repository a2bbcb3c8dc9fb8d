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


@pytest.mark.parametrize("kn", [32, 33])
def test_full_list_with_spheres_just_beyond_it(kn, gpu_lib, oracle_lib):
    """A sphere with exactly as many partners within the skin as its list holds
    and eight more a micrometre beyond, inside the margin of the float test
    (2e-6 m at these coordinates): the list is not out of room."""
    from parmec_gb300.engine import GpuEngine
    from parmec_gb300.model import Model
    from oracle.pyoracle import OracleEngine
    R, r, skin, c = 0.05, 0.01, 0.003, np.array([2.0, 2.0, 2.0])
    n = kn + 8
    k = np.arange(n) + 0.5
    th, ph = np.arccos(1.0 - 2.0 * k / n), np.pi * (1.0 + 5.0 ** 0.5) * k
    u = np.stack([np.cos(ph) * np.sin(th), np.sin(ph) * np.sin(th), np.cos(th)], -1)
    dist = np.where(np.arange(n) % 5 == 4, R + r + skin + 1e-6, R + r + 0.5 * skin)
    assert (dist > R + r + skin).sum() == 8
    out = []
    for eng in (GpuEngine(skin=skin, capacity=(kn, 32)), OracleEngine()):
        m = Model()
        mat = m.material(2500.0, 1e9, 0.25)
        m.spheres(np.concatenate([c[None], c + u * dist[:, None]]), np.array([R] + [r] * n), mat, 1)
        m.granular(0, 0, 1e6, 0.2, 0.5)
        dt = 1e-6
        m.dem(3 * dt, dt, interval=1e9, engine=eng)
        if isinstance(eng, GpuEngine):
            assert eng.diagnostics()["max_candidates"] == kn
        out.append(m)
    assert_bitwise(*out)
    assert_spheres_bitwise(*out)


@pytest.mark.parametrize("kn", [32, 64])
@pytest.mark.parametrize("n", [7, 8, 9, 15, 16, 17, 400])
def test_crowded_cells_bitwise(n, kn, gpu_lib, oracle_lib):
    """n small spheres in the few cells that a large one sets, rebuilt often,
    on both sides of the count above which the search walks one cell after
    another and of its eights."""
    from parmec_gb300.engine import GpuEngine
    from parmec_gb300.model import Model
    from oracle.pyoracle import OracleEngine
    out = []
    for eng in (GpuEngine(skin=4e-6, capacity=(kn, 64)), OracleEngine()):
        rng = np.random.default_rng(n)
        m = Model()
        mat = m.material(2500.0, 1e9, 0.25)
        g = np.stack(np.meshgrid(*(np.arange(8),) * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
        m.spheres(0.05 + g * 2.01e-3 + rng.uniform(-4e-6, 4e-6, size=(n, 3)), np.full(n, 1e-3), mat, 1)
        m.sphere((0.05 - 0.0111, 0.052, 0.052), 0.01, mat, 1)
        m.P.linear[:, :n] = rng.normal(0.0, 0.5, size=(3, n))
        m.granular(0, 0, 1e4, 0.2, 0.5)
        m.set_gravity(0.0, 0.0, -9.81)
        m.dem(59.5 * 2e-6, 2e-6, interval=1e9, engine=eng)
        if isinstance(eng, GpuEngine):
            assert eng.diagnostics()["rebuilds"] > 10 and len(eng.contacts()["mpart"]) > 0
        out.append(m)
    assert_bitwise(*out)
    assert_spheres_bitwise(*out)


@pytest.mark.parametrize("kn", [32, 33])
def test_full_list_with_triangles_bitwise(kn, gpu_lib, oracle_lib):
    """The same with a floor of triangles beside the spheres, so that the last
    places of a full list hold triangles: what is left must be in order, with
    the contacts' state in place."""
    from parmec_gb300.engine import GpuEngine
    from parmec_gb300.model import Model
    from parmec_gb300.scenes import box_triangles
    from oracle.pyoracle import OracleEngine
    R, r, skin, c = 0.05, 0.01, 3e-4, np.array([2.0, 2.0, 2.0])
    n = kn - 2 + 6                                       # two triangles of the floor, six spheres too many
    k = np.arange(n) + 0.5
    th, ph = np.arccos(1.0 - 1.5 * k / n), np.pi * (1.0 + 5.0 ** 0.5) * k
    u = np.stack([np.cos(ph) * np.sin(th), np.sin(ph) * np.sin(th), np.cos(th)], -1)
    dist = np.where(np.arange(n) % 6 == 5, R + r + skin + 1e-6, R + r - 1e-5)
    dist[np.flatnonzero(np.arange(n) % 6 == 5)[6:]] = R + r - 1e-5
    assert (dist > R + r + skin).sum() == 6
    z = 2.0 - R - 1e-4
    out = []
    for eng in (GpuEngine(skin=skin, capacity=(kn, 32)), OracleEngine()):
        m = Model()
        mat = m.material(2500.0, 1e9, 0.25)
        m.spheres(np.concatenate([c[None], c + u * dist[:, None]]), np.array([R] + [r] * n), mat, 1)
        m.obstacle([t for t in box_triangles((1.5, 1.5, z - 0.1), (2.5, 2.5, z)) if t[2] == t[5] == t[8] == z], 2)
        m.P.linear[:, 1:n + 1] = np.where(dist > R + r + skin, 0.05, 0.0) * u.T      # they never come within
        m.granular(0, 0, 1e5, 0.2, 0.5)
        dt = 2e-5
        m.dem(400.5 * dt, dt, interval=1e9, engine=eng)
        if isinstance(eng, GpuEngine):
            d = eng.diagnostics()
            assert d["max_triangles"] >= 2 and d["rebuilds"] >= 2
        out.append(m)
    assert_bitwise(*out)
    assert_spheres_bitwise(*out)
