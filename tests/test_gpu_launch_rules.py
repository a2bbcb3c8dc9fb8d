"""Both sides of the lines at which a step changes its kernels, on the GPU.

* FP64 form: up to 4,864, 9,728 and 19,456 spheres a warp tests and evaluates
  8, 16 and 32 spheres in one launch, above that two passes do; up to 19,456
  particles four lanes take a particle in the update, above that one thread.
  Adaptive steps sum the master sides in the update up to the same line.
* The commands whose scenes elsewhere in the tests are small (prescribed
  motion, restraints, body forces, torsion springs, bodies that are not
  isotropic) beside enough free spheres to take the other form.
* Mixed form: one launch for the contacts up to 38,912 spheres, two above.
* Scene gravities with 0 to 8 sine components.

FP64 states equal the oracle's bit for bit.  The mixed form is compared with
FP64 within its stated tolerances (2e-7 of the scene's size after 200 steps of
fast collisions; 20 steps here).  The device's sines differ from the host's in
the last bits: a velocity after N steps of h then differs by at most
N h times the summed amplitudes times some 1e-14 (argument and sine), checked
at 1e-12.
"""
import math
import os

import numpy as np
import pytest

from helpers import assert_bitwise, assert_spheres_bitwise, make_collision_scene

pytestmark = pytest.mark.gpu

THREADS = os.cpu_count() or 1


def cloud(n, seed=5):
    """n jittered spheres with fast random velocities and spins in a box whose
    walls move: contacts form and break within a few steps."""
    from parmec_gb300.scenes import box_triangles, critical_step
    from parmec_gb300.model import Model
    rng = np.random.default_rng(seed)
    side = math.ceil(n ** (1.0 / 3.0))
    m = Model()
    mat = m.material(2500.0, 1e9, 0.25)
    g = np.stack(np.meshgrid(*(np.arange(side),) * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    m.spheres(0.1 + g * 0.034 + rng.uniform(-0.004, 0.004, size=(n, 3)), rng.uniform(0.012, 0.02, size=n), mat, 1)
    m.P.linear[:, :n] = rng.normal(0.0, 0.5, size=(3, n))
    w = rng.normal(0.0, 5.0, size=(3, n)) * (rng.uniform(size=n) < 0.5)    # half of them not turning
    m.P.angular[0:3, :n] = w
    m.P.angular[3:6, :n] = w
    hi = 0.2 + side * 0.034
    m.obstacle(box_triangles((0.0, 0.0, 0.0), (hi, hi, hi)), 2, point=(0.5 * hi, 0.5 * hi, 0.5 * hi),
               linear=lambda t: (0.0, 0.0, 0.3), angular=lambda t: (0.0, 2.0, 1.0))
    m.granular(0, 0, 1e6, 0.2, 0.5)
    m.set_gravity(0.0, 0.0, -9.81)
    return m, 0.1 * critical_step(1e6, (4.0 / 3.0) * np.pi * 0.012 ** 3 * 2500.0, 0.2), hi


def pair(make, steps, adaptive=0.0):
    from oracle.pyoracle import OracleEngine
    from parmec_gb300.engine import GpuEngine
    out = []
    for eng in (GpuEngine(), OracleEngine(threads=THREADS)):
        m, dt = make()
        m.dem(steps * dt - 0.5 * dt, dt, interval=1e9, adaptive=adaptive, engine=eng)
        out.append(m)
    return out


@pytest.mark.parametrize("n", [1, 7, 8, 9, 33, 4864, 4865, 9728, 9729, 19456, 19457])
def test_sphere_counts_bitwise(n, gpu_lib, oracle_lib):
    mg, mo = pair(lambda: cloud(n)[:2], 20)
    assert_bitwise(mg, mo)
    assert_spheres_bitwise(mg, mo)


@pytest.mark.parametrize("n", [9, 2049, 19456, 19457])
def test_sphere_counts_adaptive_bitwise(n, gpu_lib, oracle_lib):
    mg, mo = pair(lambda: cloud(n)[:2], 1, adaptive=0.5)       # the steps it chooses are far shorter
    assert mg.curstep == mo.curstep and mg.curtime == mo.curtime
    assert_bitwise(mg, mo)
    assert_spheres_bitwise(mg, mo)


def free_spheres(m, mat, n):
    g = np.stack(np.meshgrid(*(np.arange(math.ceil(n ** (1.0 / 3.0))),) * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    if n:
        m.spheres(3.0 + 0.05 * g, np.full(n, 0.01), mat, 1)


@pytest.mark.parametrize("adaptive", [0.0, 0.5])
@pytest.mark.parametrize("pad", [0, 19457])
def test_commands_in_both_updates_bitwise(pad, adaptive, gpu_lib, oracle_lib):
    def make():
        m, dt = make_collision_scene(n_side=4, seed=4)
        body = m.analytical([1.0, 2.0, 3.0, 0.1, 0.2, -0.1], 5.0, position=(2.0, 2.0, 2.0))
        m.velocity(body, linear=(0.1, 0.2, 0.3), angular=(3.0, -2.0, 1.0))
        ts = m.tseries([0.0, 0.0, 1e-3, 0.5, 1.0, 0.5])
        m.prescribe_motion(0, linear=lambda t: (0.1, 0.0, math.sin(100 * t)), kind="vv")
        m.prescribe_motion(5, angular=lambda t: (0.0, 3.0, 0.0), kind="va")
        m.prescribe_motion(9, linear=(ts, ts, ts), angular=(ts, ts, ts), kind="aa")
        m.prescribe_motion(13, linear=lambda t: (0.0, -2.0, 0.0), angular=(ts, ts, ts), kind="av")
        m.restrain(20, linear=[0.0, 1.0, 1.0], angular=[1.0, 0.0, 0.0, 0.0, 0.0, 1.0])
        m.restrain(21, angular=[1.0, 1.0, 1.0])
        m.set_body_force(3, force=(0.5, -0.2, 1.0), torque=(0.0, 1e-3, 0.0))
        m.set_damping((0.1, 0.2, 0.3), (0.3, 0.2, 0.1))
        free_spheres(m, 0, pad)
        return m, dt
    mg, mo = pair(make, 2 if adaptive else 15, adaptive)
    assert mg.curstep == mo.curstep
    assert_bitwise(mg, mo)


@pytest.mark.parametrize("pad", [0, 19457])
def test_torsion_in_both_updates_bitwise(pad, gpu_lib, oracle_lib):
    from test_torsion import one

    def make():
        m, p, q, _ = one(10, True)
        m.spring(p, (0.5, 0.5, 0.5), q, (0.5, 0.5, 1.5), [-1.0, -1e5, 1.0, 1e5])
        free_spheres(m, 0, pad)
        return m, 1e-3
    mg, mo = pair(make, 20)
    assert_bitwise(mg, mo)


@pytest.mark.parametrize("n", [33, 38912, 38913])
def test_mixed_sphere_counts(n, gpu_lib):
    from parmec_gb300 import abi
    from parmec_gb300.engine import GpuEngine
    out = []
    for form in (abi.PG_FORM_FP64, abi.PG_FORM_MIXED):
        m, dt, hi = cloud(n)
        m.dem(20 * dt - 0.5 * dt, dt, interval=1e9, engine=GpuEngine(form=form))
        out.append(m)
    a, b = out
    assert np.max(np.abs(a.P.position[0:3, :n] - b.P.position[0:3, :n])) <= 2e-7 * hi
    fa, fb = a.P.force[:, :n], b.P.force[:, :n]
    assert np.max(np.abs(fa - fb)) <= 1e-3 * np.max(np.abs(fa))


@pytest.mark.parametrize("form", [0, 1])
@pytest.mark.parametrize("ncomp", [0, 1, 3, 7, 8])
def test_excitation_components(ncomp, form, gpu_lib):
    from parmec_gb300 import batch
    from parmec_gb300.engine import GpuEngine
    from parmec_gb300.model import Model
    from parmec_gb300.serving import excitation_gravity
    comps = [(1.0 + k, 3.0 + 5.0 * k, 0.1 * k) for k in range(ncomp)]
    excs = [batch.excitation((0.0, 0.5, -9.81), (0.6, 0.0, 0.8), comps), batch.excitation((1.0, 0.0, 0.0), (0.0, 1.0, 0.0), comps)]
    models = []
    for _ in excs:
        m = Model()
        m.sphere((0.0, 0.0, 0.0), 0.1, m.material(1000.0, 1e9, 0.25), 1)
        m.granular(0, 0, 1e6, 0.2, 0.5)
        models.append(m)
    P, _ = batch.pool(models)
    eng = GpuEngine(form=form)
    eng.attach(P)
    for k, exc in enumerate(excs):
        eng.set_scene(k, True, excitation=exc, start=0)
    P.engine = eng
    P._dirty = False
    dt, steps = 1e-3, 50
    P.dem(steps * dt - 0.5 * dt, dt, interval=1e9, engine=eng)
    for k, exc in enumerate(excs):
        batch.extract(P, k, models[k])
        g = excitation_gravity(exc)
        want = dt * np.sum([g(s * dt) for s in range(steps)], axis=0)
        scale = steps * dt * (10.0 + sum(a for a, _, _ in comps))
        tol = 1e-12 if form == 0 else 4 * 2.0 ** -24
        assert np.max(np.abs(models[k].P.linear[:, 0] - want)) <= tol * scale
    eng.close()
