"""The choice of the Euler element stage, fixed point or FP64, at p = 1..4."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu
OPEN = (-4, -4, -4, -4)


def riemann(dg, p, limiter):
    mesh = dg.Mesh.square(13, 11, jitter=0.1, seed=3, bc=OPEN)
    s = dg.Solver(mesh, dg.EULER, p, problem="euler_riemann4", limiter=limiter, cfl=0.2)
    s.init_conditions()
    return s


@pytest.mark.parametrize("limiter", [0, 1])
@pytest.mark.parametrize("p", [1, 2, 3, 4])
def test_what_is_switched_on_or_off_runs(dglib, p, limiter):
    """Both stages can be chosen at every order, and are two: they agree to
    rounding and not in their bits.  A solver left alone runs the fixed-point one."""
    dg = dglib
    on, off, default = (riemann(dg, p, limiter) for _ in range(3))
    on.tensor_contractions = True
    off.tensor_contractions = False
    assert on.tensor_contractions and not off.tensor_contractions
    assert (on.element_stage, off.element_stage, default.element_stage) == (2, 1, 2)
    for s in (on, off, default):
        s.step(6, dg.SSP_RK3, 0.0)
    a, b = on.get_state(), off.get_state()
    assert relerr(a, b, 4) <= 1e-12 and not np.array_equal(a, b)
    assert np.array_equal(default.get_state(), a)


def test_the_autotuner_reports_and_leaves_the_stage_that_runs(dglib):
    dg = dglib
    s = riemann(dg, 1, 1)
    _, stage = s.autotune_stage()
    assert s.element_stage == stage and s.tensor_contractions == (stage == 2)
