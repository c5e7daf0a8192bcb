"""The limiter on states with infinities and NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
OPEN = (-4, -4, -4, -4)
MEAN = {0: (1.0,), 1: (1.0, 0.3, -0.2, 2.5), 2: (1.0, 0.1, -0.2), 3: (0.4, -0.3, 0.5)}


def uniform(dg, eq, p):
    """A solver with the limiter on and a uniform state: every bound collapses
    to the mean."""
    mesh = dg.Mesh.square(6, 5, jitter=0.1, seed=2, bc=OPEN)
    s = dg.Solver(mesh, eq, p, limiter=1, cfl=0.1)
    c = np.zeros(s.shape)
    c[:, 0, :] = np.array(MEAN[eq])[:, None]
    return s, c


@pytest.mark.parametrize("fixed", [True, False])
@pytest.mark.parametrize("eq", [0, 1, 2, 3])
@pytest.mark.parametrize("p", [2, 3, 4])
def test_a_nan_is_not_limited_away(dglib, eq, p, fixed):
    dg = dglib
    s, c = uniform(dg, eq, p)
    if eq == dg.EULER:
        s.tensor_contractions = fixed
    elif not fixed:
        pytest.skip("one element stage")
    for bad in (np.nan, -np.nan):
        d = c.copy()
        d[0, 3, 17] = bad
        s.set_state(d)
        s.limit_c()
        assert np.array_equal(s.get_state(), d, equal_nan=True)
        # nor where a run from a new state limits and traces it in one pass (a depth
        # that is not a number is not physical: the positivity rule flattens it)
        if eq == dg.SHALLOW_WATER:
            continue
        s.set_state(d)
        s.step(1, dg.SSP_RK3, 0.0)
        assert not np.isfinite(s.get_state()[0, :, 17]).all()


@pytest.mark.parametrize("eq", [0, 1, 2, 3])
@pytest.mark.parametrize("p", [2, 3, 4])
def test_an_infinity_is_an_overshoot_like_any_other(dglib, eq, p):
    dg = dglib
    s, c = uniform(dg, eq, p)
    d = c.copy()
    d[0, 3, 17] = np.inf
    s.set_state(d)
    s.limit_c()
    assert np.array_equal(s.get_state(), c)
