"""The limiter: its quotients, and states with infinities and NaN."""
import numpy as np
import pytest

from conftest import ref_tables, split_tables

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


@pytest.mark.parametrize("eq", [0, 1, 2, 3])
def test_alpha_is_the_smaller_ieee_quotient(dglib, eq):
    """Tables and states of a few bits, so that traces, bounds and overshoots
    are exact: the limited slopes are those of IEEE division and
    multiplication, bit for bit."""
    dg = dglib
    mesh = dg.Mesh.square(12, 11, jitter=0.1, seed=2)
    s = dg.Solver(mesh, eq, 1, limiter=1)
    tab = [t.copy() for t in split_tables(ref_tables(1), 1)]
    tab[0][:3] = 1.0  # phi_0 = 1 at the area points
    E = np.array([[[1.0, 0.5, -0.25], [1.0, 0.25, 1.0]], [[1.0, -0.5, 0.25], [1.0, -1.0, 0.5]],
                  [[1.0, 0.125, -1.0], [1.0, -0.25, -0.5]]])  # [face][point][mode]
    tab[3][:] = E.transpose(0, 2, 1).ravel()
    s.set_tables(*tab)
    if eq == dg.EULER:
        s.tensor_contractions = True
    rng = np.random.default_rng(eq)
    c = np.round(rng.uniform(-1, 1, s.shape) * 2.0 ** 20) / 2.0 ** 20
    c[:, 0] *= 0.25
    s.set_state(c)
    s.limit_c()
    _, es, _, se = mesh.arrays()
    nb = np.array([[se[1, sd] if se[0, sd] == e else se[0, sd] for sd in es[:, e]]
                   for e in range(s.K)])
    ref, limited = c.copy(), 0
    for n in range(s.N):
        for e in range(s.K):
            m = c[n, 0, [e] + list(nb[e])]
            T = np.einsum("fji,i->fj", E, c[n, :, e])
            up, dn = T.max() - m[0], m[0] - T.min()
            lo, hi = m[0] - m.min(), m.max() - m[0]
            al = min(lo / up if up > lo else 1.0, hi / dn if dn > hi else 1.0)
            if al < 1:
                limited += 1
                ref[n, 1:, e] *= al
    assert limited > s.N * s.K // 2
    assert np.array_equal(s.get_state(), ref)


@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("eq", [1, 2])
def test_a_flattened_state_steps_as_its_means_do(dglib, eq, p):
    """Elements whose traces are not physical are flattened to their means: a
    run from the state is the run from the flattened one, bit for bit."""
    dg = dglib
    mesh = dg.Mesh.square(7, 6, jitter=0.1, seed=2, bc=OPEN)
    s, f = (dg.Solver(mesh, eq, p, cfl=0.1, gravity=9.81) for _ in range(2))
    if eq == dg.EULER:
        s.tensor_contractions = f.tensor_contractions = True
    rng = np.random.default_rng(p)
    c = 0.01 * rng.standard_normal(s.shape)
    c[:, 0, :] += np.array(MEAN[eq])[:, None] * (1 + 0.2 * rng.standard_normal((s.N, s.K)))
    c[0, 1:, ::2] *= 400  # a negative density or depth on some edge
    d = c.copy()
    d[:, 1:, ::2] = 0
    s.set_state(c)
    f.set_state(d)
    assert s.step(1, dg.SSP_RK3, 0.0) == f.step(1, dg.SSP_RK3, 0.0)
    assert np.array_equal(s.get_state(), f.get_state())


@pytest.mark.parametrize("p", [2, 3, 4, 5])
@pytest.mark.parametrize("eq", [0, 2, 3])
def test_a_run_goes_on_from_a_limited_state_as_a_new_one_does(dglib, eq, p):
    """The traces a limited stage leaves are those a new run forms: where
    limiting the state again changes nothing, the next step's bits agree."""
    dg = dglib
    checked = 0
    for seed in range(60):
        mesh = dg.Mesh.square(1, 1, jitter=0.0, seed=1, bc=OPEN)
        s, f = (dg.Solver(mesh, eq, p, limiter=1, cfl=0.1, gravity=9.81) for _ in range(2))
        rng = np.random.default_rng(seed)
        c = 0.1 * rng.standard_normal(s.shape)
        c[:, 0, :] += np.array(MEAN[eq])[:, None]
        s.set_state(c)
        t = s.step(1, dg.SSP_RK3, 0.0)
        u = s.get_state()
        f.set_state(u)
        f.limit_c()
        if not np.array_equal(f.get_state(), u):
            continue
        checked += 1
        assert s.step(1, dg.SSP_RK3, t) == f.step(1, dg.SSP_RK3, t)
        assert np.array_equal(s.get_state(), f.get_state())
    assert checked >= 5
