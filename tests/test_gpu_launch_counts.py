"""The session's count of its kernel launches: of a run through CUDA graphs it
is the kernels in them, of one without it is what the launch rules say.  Both
must agree on either side of the lines at which a step changes its kernels."""
import pytest

from test_gpu_launch_rules import cloud

pytestmark = pytest.mark.gpu


def counts(make, steps, adaptive=0.0, form=0):
    from parmec_gb300.engine import GpuEngine
    out = []
    for graph in (True, False):
        m, dt = make()
        eng = GpuEngine(form=form, graph=graph)
        m.dem(steps * dt - 0.5 * dt, dt, interval=1e9, adaptive=adaptive, engine=eng)
        out.append((eng.kernel_launches(), m.curstep if adaptive else 0))
        eng.close()
    return out


@pytest.mark.parametrize("n", [33, 19455, 19456, 19457, 97000, 100000])
def test_fixed_steps(n, gpu_lib):
    """19,456 particles and a block of obstacles are one block more than the
    wave in which the update ends the step; 97,000 fill it with 128 a block."""
    a, b = counts(lambda: cloud(n)[:2], 9)
    assert a == b


@pytest.mark.parametrize("n", [9, 19455, 19456, 19457])
def test_adaptive_steps(n, gpu_lib):
    a, b = counts(lambda: cloud(n)[:2], 1, adaptive=0.5)
    assert a == b


@pytest.mark.parametrize("n", [33, 38912, 38913, 160000])
def test_mixed_form(n, gpu_lib):
    a, b = counts(lambda: cloud(n)[:2], 9, form=1)
    assert a == b


@pytest.mark.parametrize("adaptive", [0.0, 0.5])
def test_springs_without_spheres(adaptive, gpu_lib):
    from parmec_gb300.scenes import spring_lattice
    a, b = counts(lambda: spring_lattice(12), 3, adaptive=adaptive)
    assert a == b
