"""Basis tables handed to a solver (dg_solver_set_tables)."""
import numpy as np
import pytest

from conftest import ref_tables, relerr, split_tables

pytestmark = pytest.mark.gpu
HUMP = (1.0, 0.1, 0.1, 0.45, 0.55)


@pytest.mark.parametrize("p", [1, 2, 3, 4])
def test_tables_set_after_a_bed_rebuild_its_slopes(dglib, oracle_mod, p):
    """Tables whose slope entries are scaled change the bed's source with the
    rest of the operator: the oracle's with the same tables, whichever of bed
    and tables came first."""
    dg = dglib
    mesh = dg.Mesh.square(6, 5, jitter=0.1, seed=3, bc=(-1, -1, -1, -1))
    tab = split_tables(ref_tables(p), p)
    for k in (1, 2):
        tab[k] = tab[k] * 1.25
    o = oracle_mod.Oracle.from_mesh(mesh, dg.SHALLOW_WATER, p,
                                    oracle_mod.prm_vec(g=9.81, extra=HUMP),
                                    dg.PROBLEMS["sw_hump"])
    out = []
    for first in (True, False):
        s = dg.Solver(mesh, dg.SHALLOW_WATER, p, problem="sw_hump", prm=HUMP, gravity=9.81)
        s.init_conditions()
        c = s.get_state()
        if first:
            s.bathymetry_project("sine", (0.1, 1.0, 1.0))
            b = s.get_bathymetry()
        s.eval_rhs(c, 0.0)
        s.set_tables(*tab)
        if not first:
            s.set_bathymetry(b)
        out.append(s.eval_rhs(c, 0.0))
    o.set_tables(np.concatenate(tab))
    o.set_bathymetry(b)
    assert np.array_equal(out[0], out[1])
    assert relerr(out[0], o.rhs(c, 0.0), 3) <= 1e-12


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_tables_that_are_not_finite_are_refused(dglib, bad):
    """And leave the tables before them."""
    dg = dglib
    mesh = dg.Mesh.square(4, 4, jitter=0.1, seed=3)
    s = dg.Solver(mesh, dg.ADVECTION, 2, problem="adv_sine")
    s.init_conditions()
    c = s.get_state()
    r = s.eval_rhs(c, 0.0)
    for k in range(4):  # values, both slopes, edge values
        tab = split_tables(ref_tables(2), 2)
        tab[k] = tab[k].copy()
        tab[k][-1] = bad
        with pytest.raises(dg.DGError):
            s.set_tables(*tab)
    assert np.array_equal(s.eval_rhs(c, 0.0), r)
