"""The mesh contact's pair list where it changes: room, searches, far places.

Every comparison is with the oracle's brute-force search, bit for bit.
"""
import ctypes

import numpy as np
import pytest

from helpers import assert_bitwise

pytestmark = pytest.mark.gpu

DT = 1e-5


def pile(origin=(0.0, 0.0, 0.0), layers=2, side=3, seed=3, radius=1e-3, first=0.0021, gap=0.0021):
    """Layers of 10 mm cubes over a fixed plate (`first` and `gap` above what
    lies below, 0.1 mm outside the reach), the upper ones turning and falling
    at 1 m/s.  The pile
    is made near zero and moved to its origin (the volume integrals of a MESH
    lose a small body's inertia far away)."""
    from parmec_gb300 import mesh
    from parmec_gb300.model import Model
    rng = np.random.default_rng(seed)
    m = Model()
    mat = m.material(2500.0, 1e9, 0.25)
    lo, hi = (-0.01, -0.01, -0.005), (0.014 * side, 0.014 * side, 0.0)
    c = [(x, y, z) for z in (lo[2], hi[2]) for x, y in ((lo[0], lo[1]), (hi[0], lo[1]), (hi[0], hi[1]), (lo[0], hi[1]))]
    plate = m.mesh([v for p in c for v in p], [8, 0, 1, 2, 3, 4, 5, 6, 7, mat], mat, 2)
    m.prescribe_motion(plate, linear=lambda t: (0.0, 0.0, 0.0), angular=lambda t: (0.0, 0.0, 0.0), kind="vv")
    org = [(0.014 * i + 1e-3 * rng.uniform(-1, 1), 0.014 * j, first + (0.01 + gap) * k)
           for k in range(layers) for i in range(side) for j in range(side)]
    parts = mesh.hex_grid(m, np.array(org), 0.01, mat, 1)
    for p in parts[side * side:]:
        m.velocity(int(p), linear=(0.0, 0.0, -1.0), angular=tuple(float(x) for x in rng.normal(0.0, 2.0, size=3)))
    m.granular(0, 0, 1e4, 0.3, 0.4)
    m.set_gravity(0.0, 0.0, -9.81)
    m.mesh_contact(radius)
    for c in range(3):
        m.P.position[[c, 3 + c], :m.parnum] += origin[c]
        m.N.nodes[[c, 3 + c], :m.nodnum] += origin[c]
        m.Tr.tri[[c, 3 + c, 6 + c], :m.trinum] += origin[c]
    return m


def pair(make):
    from oracle.pyoracle import OracleEngine
    from parmec_gb300.engine import GpuEngine
    return (make(), GpuEngine()), (make(), OracleEngine())


def dem(both, steps, first=False):
    for m, eng in both:
        m.dem((steps - (0.5 if first else 0.0)) * DT, DT, interval=1e9, engine=eng)
    assert_bitwise(both[0][0], both[1][0])
    assert both[0][1].mesh_contact_stats() == both[1][1].mesh_contact_stats()
    return both[1][1].mesh_contact_stats()


def test_refused_list_ends_the_run_and_the_session_goes_on(gpu_lib, oracle_lib):
    """A search that finds more pairs than there is room for ends the run with
    an error, at the step it belongs to; with room again the session goes on
    from there, its contacts' state unbroken."""
    from parmec_gb300 import abi, driver
    both = (mg, eg), _ = pair(pile)
    assert dem(both, 300, first=True)[1] > 0
    tabs = driver.StepTables(mg, [mg.curtime + k * DT for k in range(400)], DT, [1e9, 1e9], [None, None], [-1, -1])
    done0 = eg.global_step()
    assert eg.lib.pg_session_mesh_contact_room(eg.sess, 1, 0, 0) == abi.PG_OK
    tab = tabs.ctab(0, 400)
    assert eg.lib.pg_session_run(eg.sess, ctypes.byref(tab), DT) == abi.PG_ERR_CAPACITY
    done = eg.global_step() - done0
    assert 0 < done < 400
    assert eg.lib.pg_session_run(eg.sess, ctypes.byref(tab), DT) == abi.PG_ERR_CAPACITY
    assert eg.global_step() == done0 + done
    assert eg.lib.pg_session_mesh_contact_room(eg.sess, 0, 0, 0) == abi.PG_OK
    tab = tabs.ctab(done, 400)
    assert eg.lib.pg_session_run(eg.sess, ctypes.byref(tab), DT) == abi.PG_OK
    eg.download()
    mo, eo = both[1]
    mo.dem(400 * DT, DT, interval=1e9, engine=eo)
    assert_bitwise(mg, mo)
    assert eg.mesh_contact_stats() == eo.mesh_contact_stats()


@pytest.mark.parametrize("origin", [(0.0, 0.0, 0.0), (3e5, -3e5, 1e4)])
def test_pile_far_from_the_origin_bitwise(origin, gpu_lib, oracle_lib):
    """Searches while the upper layer falls, near the origin and where a
    georeferenced scene lies."""
    both = pair(lambda: pile(origin))
    dem(both, 100, first=True)
    assert dem(both, 300)[1] > 20


def test_boxes_far_from_the_origin_find_no_more_pairs(gpu_lib):
    """A 5 x 5 x 5 stack of 10 mm cubes 1 mm apart, reach 0.2 mm: no pair,
    wherever it stands."""
    from parmec_gb300 import mesh
    from parmec_gb300.engine import GpuEngine
    from parmec_gb300.model import Model
    for x in (0.0, 1e4, 3e5):
        m = Model()
        mat = m.material(2500.0, 1e9, 0.25)
        g = np.stack(np.meshgrid(*(np.arange(5),) * 3, indexing="ij"), -1).reshape(-1, 3)
        mesh.hex_grid(m, x + 0.011 * g, 0.01, mat, 1)
        m.granular(0, 0, 1e5, 0.3, 0.4)
        m.mesh_contact(1e-4)
        eng = GpuEngine()
        m.dem(2 * DT, DT, interval=1e9, engine=eng)
        assert eng.mesh_contact_stats() == (0, 0)
        eng.close()


def test_more_partners_in_the_skin_than_a_list_holds(gpu_lib, oracle_lib):
    """Cubes in a grid of cells a hundred times their size: the skin, a part of
    the cell, reaches more triangles than a list holds, the swept boxes do not."""
    from parmec_gb300 import abi
    from parmec_gb300.mesh import mesh_contact_grid
    both = (mg, eg), _ = pair(lambda: pile(layers=3))
    eg.attach(mg)
    mg.engine, mg._dirty = eg, False
    cell, big = mesh_contact_grid(mg)
    assert 27 * 12 - 12 > 256 and 0.5 * cell > 0.0021
    assert eg.lib.pg_session_mesh_contact(eg.sess, 1e-3, 100.0 * cell, big.ctypes.data) == abi.PG_OK
    dem(both, 30, first=True)
    assert dem(both, 100)[1] > 20


def test_pair_arrays_grow_with_contacts_carried(gpu_lib, oracle_lib):
    """36 cubes resting on the plate when as many fall on them: the list
    outgrows its arrays while contacts hold tangential state."""
    both = pair(lambda: pile(side=6, first=0.0019, gap=0.0025))
    few = dem(both, 20, first=True)
    many = dem(both, 60)
    assert few[1] >= 36 and many[0] > 1.5 * (1.5 * few[0] + 1024)


@pytest.mark.parametrize("vertex,edge", [(37, 0), (0, 37), (37, 37), (1, 1)])
def test_distances_without_room_bitwise(vertex, edge, gpu_lib, oracle_lib):
    """Near pairs that find no room for their distances, in either list or in
    both, take the whole narrow phase: the same bits."""
    from parmec_gb300 import abi
    both = (mg, eg), _ = pair(pile)
    eg.attach(mg)
    mg.engine, mg._dirty = eg, False
    assert eg.lib.pg_session_mesh_contact_room(eg.sess, 0, vertex, edge) == abi.PG_OK
    dem(both, 60, first=True)
    assert dem(both, 100)[1] > 37


def test_fast_meshes_bitwise(gpu_lib, oracle_lib):
    """A pile whose upper layer flies past and into the lower one at 20 m/s, so
    that the skin grows, then slowed down, so that it shrinks again."""
    both = pair(lambda: pile(gap=0.004))
    for m, _ in both:
        m.P.linear[:, 10:m.parnum] = np.array([[20.0], [3.0], [-5.0]])
    dem(both, 60, first=True)
    assert dem(both, 60)[1] > 0
    for m, _ in both:
        m.P.linear[:, 1:m.parnum] *= 0.02
        m.P.angular[:, 1:m.parnum] *= 0.02
        m._dirty = True
    dem(both, 150)
    dem(both, 300)
