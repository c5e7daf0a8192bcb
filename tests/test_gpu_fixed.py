"""The element stage's fixed-point contractions (dg_fixed.cuh): every equation
and order at the edges of its 32-element tiles against the oracle, rows at
the ends of the double range, zeros and non-finite entries."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu

RHS_TOL = 1e-12  # the right-hand side's parity bound (test_gpu_parity.py)
OPEN = (-4, -4, -4, -4)


def random_state(s, seed, amp=0.02):
    """Means that every equation takes as physical, small higher modes."""
    rng = np.random.default_rng(seed)
    c = np.zeros(s.shape)
    mean = {0: (1.0,), 1: (1.0, 0.3, -0.2, 2.5), 2: (1.0, 0.1, -0.2), 3: (0.4, -0.3, 0.5)}[s.eq]
    c[:, 0, :] = np.array(mean)[:, None] * (1 + 0.1 * rng.standard_normal((s.N, s.K)))
    c[:, 1:, :] = amp * rng.standard_normal((s.N, s.n_p - 1, s.K))
    return c


def problem(dg, eq, p, nx, ny, bc=OPEN, seed=2):
    mesh = dg.Mesh.square(nx, ny, jitter=0.1, seed=seed, bc=bc)
    return mesh, dg.Solver(mesh, eq, p, gravity=9.81)


@pytest.mark.parametrize("nx,ny", [(1, 1), (4, 4), (3, 11)])  # 2, 32 and 66 elements
@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("eq", [0, 1, 2, 3])
def test_rhs_matches_oracle_at_tile_edges(dglib, oracle_mod, eq, p, nx, ny):
    dg = dglib
    mesh, s = problem(dg, eq, p, nx, ny)
    if eq == dg.EULER:
        s.tensor_contractions = True
    o = oracle_mod.Oracle.from_mesh(mesh, eq, p, oracle_mod.prm_vec(g=9.81), 0)
    if eq == dg.SHALLOW_WATER:
        s.bathymetry_project("sine", (0.1, 1.0, 1.0))
        o.set_bathymetry(s.get_bathymetry())
    c = random_state(s, 10 * eq + p)
    assert relerr(s.eval_rhs(c, 0.0), o.rhs(c, 0.0), s.N) <= RHS_TOL


@pytest.mark.parametrize("p", [1, 4])
@pytest.mark.parametrize("eq", [0, 3])
@pytest.mark.parametrize("k", [-960, 890])
def test_rows_at_the_ends_of_the_range(dglib, eq, p, k):
    """A linear operator on a state scaled by 2^k, rows whose exponents leave
    the range that is computed directly: the scaled result."""
    dg = dglib
    _, s = problem(dg, eq, p, 5, 4)
    c = random_state(s, 3)
    r = s.eval_rhs(c, 0.0)
    assert relerr(np.ldexp(s.eval_rhs(np.ldexp(c, k), 0.0), -k), r, s.N) <= RHS_TOL


@pytest.mark.parametrize("k", [-450, -260, 260, 450])
def test_face_momenta_at_the_ends_of_the_range(dglib, k):
    """The Euler flux is homogeneous of degree one: a state scaled by 2^k has
    the right-hand side scaled by 2^k, with momenta whose products stay in
    the range that the face kernel computes in fixed point (|k| = 260) and
    with such as leave it (450), and states at rest among them."""
    dg = dglib
    _, s = problem(dg, dg.EULER, 1, 5, 4)
    c = random_state(s, 5)
    c[1:3, :, ::3] = 0
    c[2, :, 1::3] = 0
    r = s.eval_rhs(c, 0.0)
    assert relerr(np.ldexp(s.eval_rhs(np.ldexp(c, k), 0.0), -k), r, s.N) <= RHS_TOL


@pytest.mark.parametrize("eq", [0, 3])
def test_zero_and_non_finite_rows(dglib, eq):
    """A zero state has a zero right-hand side; a NaN or an infinity in one
    element leaves every element that does not touch it as it is and does
    not come out of its own as a number."""
    dg = dglib
    mesh, s = problem(dg, eq, 3, 8, 8)
    assert not s.eval_rhs(np.zeros(s.shape), 0.0).any()
    c = random_state(s, 4)
    r = s.eval_rhs(c, 0.0)
    _, es, _, se = mesh.arrays()
    e = 57
    near = {e} | {int(v) for sd in es[:, e] for v in se[:2, sd] if v >= 0}
    far = np.array([k for k in range(s.K) if k not in near])
    for bad in (np.nan, np.inf):
        d = c.copy()
        d[0, 2, e] = bad
        q = s.eval_rhs(d, 0.0)
        assert np.array_equal(q[:, :, far], r[:, :, far])
        assert not np.isfinite(q[:, 1:, e]).all()


@pytest.mark.parametrize("p", [1, 3])
@pytest.mark.parametrize("eq", [1, 3])
def test_limiter_of_tiny_and_huge_states(dglib, eq, p):
    """The limiter commutes with a scaling by 2^k, also where the products of
    the bounds' distances that pick the smaller quotient leave the range."""
    dg = dglib
    mesh = dg.Mesh.square(6, 5, jitter=0.1, seed=2, bc=OPEN)
    s = dg.Solver(mesh, eq, p, limiter=1)
    c = random_state(s, 6, amp=0.2)

    def limited(k):
        s.set_state(np.ldexp(c, k))
        s.limit_c()
        return np.ldexp(s.get_state(), -k)

    r = limited(0)
    assert not np.array_equal(r, c)
    for k in (-560, 600):
        assert relerr(limited(k), r, s.N) <= RHS_TOL
