"""The numerical fluxes of the face kernels where one state is far from the
other: a wave speed that is not a number on one side only, and small
components beside large ones."""
import numpy as np
import pytest

from conftest import relerr

pytestmark = pytest.mark.gpu
OPEN = (-4, -4, -4, -4)
RHS_TOL = 1e-12  # the right-hand side's parity bound (test_gpu_parity.py)


def uniform(s, U):
    c = np.zeros(s.shape)
    c[:, 0, :] = np.array(U)[:, None] / np.sqrt(2.0)
    return c


@pytest.mark.parametrize("eq,bad", [(1, (1.0, 0.2, 0.1, -0.1)), (2, (-0.1, 0.02, 0.01))])
def test_a_sound_speed_that_is_not_a_number_gives_way_to_the_other_sides(dglib, oracle_mod, eq,
                                                                         bad):
    """An element with a negative mean pressure (depth) has no sound speed;
    its neighbours' fluxes take their own, whether it lies left or right of
    the side in the mesh's order."""
    dg = dglib
    mesh = dg.Mesh.square(5, 4, jitter=0.1, seed=2, bc=OPEN)
    s = dg.Solver(mesh, eq, 1, gravity=9.81)
    o = oracle_mod.Oracle.from_mesh(mesh, eq, 1, oracle_mod.prm_vec(g=9.81), 0)
    _, es, _, se = mesh.arrays()
    lefts = 0
    for e in range(s.K):
        if any((se[:2, sd] < 0).any() for sd in es[:, e]):
            continue  # its ghost state has none either
        c = uniform(s, (1.0, 0.3, -0.2, 2.5)[:s.N])
        c[:, 0, e] = np.array(bad) / np.sqrt(2.0)
        r = s.eval_rhs(c, 0.0)
        assert np.isfinite(r).all()
        # the oracle takes the other side's speed where the element is the left one
        left = [sd for sd in es[:, e] if se[0, sd] == e]
        for sd in left:
            k = se[1, sd]
            ref = o.rhs(c, 0.0)[:, :, k]
            if np.isfinite(ref).all():
                lefts += 1
                assert relerr(r[:, :, k], ref, s.N) <= RHS_TOL
    assert lefts > 0


@pytest.mark.parametrize("var", [1, 2])
@pytest.mark.parametrize("r", [1e-3, 1e-9, 1e-15])
def test_a_small_momentum_beside_a_large_one_keeps_its_bits(dglib, oracle_mod, var, r):
    """Flow along one axis (shallow water with next to no gravity): the
    small component's right-hand side, all of whose terms are as small, to
    the parity bound of its own norm."""
    dg = dglib
    mesh = dg.Mesh.square(6, 5, jitter=0.1, seed=4, bc=OPEN)
    s = dg.Solver(mesh, dg.SHALLOW_WATER, 2, gravity=1e-40)
    rng = np.random.default_rng(3)
    c = uniform(s, (1.0, 1.0, 1.0))
    c[:, 0, :] *= 1 + 0.2 * rng.standard_normal((3, s.K))
    c[:, 1:, :] = 0.02 * rng.standard_normal((3, s.n_p - 1, s.K))
    c[var] *= r
    o = oracle_mod.Oracle.from_mesh(mesh, dg.SHALLOW_WATER, 2, oracle_mod.prm_vec(g=1e-40), 0)
    assert relerr(s.eval_rhs(c, 0.0), o.rhs(c, 0.0), 3) <= RHS_TOL
