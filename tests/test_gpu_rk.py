"""The RK4 and midpoint RK2 loops without the limiter, whose stages form the
next one's input, its traces and RK4's sum in the element stage's epilogue:
systems at sizes that are no multiple of its 32-element tiles, and elements
that are flattened on the way, against the oracle."""
import numpy as np
import pytest

from conftest import ref_tables, relerr, split_tables

pytestmark = pytest.mark.gpu
STATE_TOL = 1e-10  # the steps' parity bound (test_gpu_steps.py)
VTX = (5.0, 5.0, 5.0, 1.0, 1.0, 10.0)
HUMP = (1.0, 0.1, 0.1, 0.45, 0.55)
CASES = {  # equation, problem, box, sides, problem parameters, bed
    "euler_vortex": (1, "euler_vortex", (0, 10, 0, 10), (0, 0, 0, 0), VTX, False),
    "shallow_water_bed": (2, "sw_hump", (0, 1, 0, 1), (-1, -1, -1, -1), HUMP, True),
    "maxwell_plane": (3, "maxwell_plane", (0, 1, 0, 1), (0, 0, 0, 0), (), False),
}


def pair(dg, oracle_mod, case, p, nx=7, ny=5):
    eq, pb, box, bc, prm, bed = CASES[case]
    mesh = dg.Mesh.square(nx, ny, box=box, jitter=0.1, seed=5, bc=bc)
    s = dg.Solver(mesh, eq, p, problem=pb, cfl=0.2, gravity=9.81, prm=prm)
    if eq == dg.EULER:
        s.tensor_contractions = True
    o = oracle_mod.Oracle.from_mesh(mesh, eq, p, oracle_mod.prm_vec(g=9.81, extra=prm),
                                    dg.PROBLEMS[pb])
    # one tabulation on both sides: at p = 4 the oracle's own differs from the
    # library's by 5e-14, which the small component of the Maxwell wave shows
    tab = ref_tables(p)
    s.set_tables(*split_tables(tab, p))
    o.set_tables(tab)
    if bed:
        s.bathymetry_project("sine", (0.1, 1.0, 1.0))
        o.set_bathymetry(s.get_bathymetry())
    s.init_conditions()
    return s, o


SCHEMES = {"RK4": 1, "RK2": 2}  # the oracle's numbers


@pytest.mark.parametrize("scheme", sorted(SCHEMES))
@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("case", sorted(CASES))
def test_systems_match_the_oracle(dglib, oracle_mod, case, p, scheme):
    dg = dglib
    s, o = pair(dg, oracle_mod, case, p)
    assert s.K % 32
    c0 = s.get_state()
    t = s.step(8, getattr(dg, scheme), 0.0)
    c, to, n = o.step(c0, 8, SCHEMES[scheme], 0, 0.2)
    assert n == 8 and abs(t - to) <= 1e-12 * to
    assert relerr(s.get_state(), c, s.N) <= STATE_TOL


def dip(p):
    """Modes of 40 (r^2 + s^2 + r s - r - s + 1/3 - 1/20): above 1 on the edges,
    negative at an area point."""
    tab = split_tables(ref_tables(p), p)
    w, r, s = tab[5:8]
    f = 40 * (r * r + s * s + r * s - r - s + 1 / 3 - 1 / 20)
    assert f.min() < 0
    return tab[0].reshape(-1, len(w)) @ (w * f)


def thin(p):
    """Modes of a gas in fast uniform flow whose density falls to a fiftieth of
    its mean at one edge point, physical everywhere."""
    tab = split_tables(ref_tables(p), p)
    n = (p + 1) * (p + 2) // 2
    least = min(tab[3].reshape(3, n, p + 1)[:, 1].min(), tab[0].reshape(n, -1)[1].min())
    rho = np.zeros(n)
    rho[:2] = 1 / np.sqrt(2), (0.02 - 1) / least
    c = np.stack([rho, -6 * rho, -3 * rho, 0.5 * 45 * rho])
    c[3, 0] += 0.2 / np.sqrt(2)
    return c


@pytest.mark.parametrize("scheme", sorted(SCHEMES))
@pytest.mark.parametrize("p", [2, 3, 4])
@pytest.mark.parametrize("where", ["area", "trace", "later"])
def test_flattened_elements_match_the_oracle(dglib, oracle_mod, p, scheme, where):
    """A density that is negative at an area point alone, and at edge points
    (which flatten before the fluxes), in the first stage's input; and one
    that becomes so in a later stage's."""
    dg = dglib
    s, o = pair(dg, oracle_mod, "euler_vortex", p)
    c0 = s.get_state()
    sel = np.arange(s.K) % 9 == 4
    if where == "area":
        c0[0][:, sel] = dip(p)[:, None]
    elif where == "trace":
        c0[0, 1, sel] = 1.2
    else:
        c0[:, :, sel] = thin(p)[:, :, None]
    o.rhs(c0, 0.0)
    assert o.flattened() == (0 if where == "later" else sel.sum())
    s.set_state(c0)
    t = s.step(1, getattr(dg, scheme), 0.0)
    c, to, n = o.step(c0, 1, SCHEMES[scheme], 0, 0.2)
    assert o.flattened() >= sel.sum()
    assert n == 1 and abs(t - to) <= 1e-12 * to
    assert relerr(s.get_state(), c, s.N) <= STATE_TOL


@pytest.mark.parametrize("scheme", ["RK4", "RK2", "SSP_RK3"])
@pytest.mark.parametrize("p", [1, 3])
@pytest.mark.parametrize("case", ["euler_vortex", "maxwell_plane"])
def test_small_increments_reach_the_state_whole(dglib, oracle_mod, case, p, scheme):
    """A time step so short that the whole increment is about an ulp of the
    state: RK4 and RK2 round the state once, to u + dt L(u), where parts added
    one after another would be lost; SSP-RK3 combines states and may be two
    roundings off."""
    dg = dglib
    s, _ = pair(dg, oracle_mod, case, p)
    c = s.get_state()
    L = s.eval_rhs(c, 0.0)
    big = np.abs(c) > 1e-3
    dt = 0.8 * np.median(np.spacing(np.abs(c[big])) / np.abs(L[big]))
    s.step(1, getattr(dg, scheme), 0.0, dt=dt)
    u, ref = s.get_state(), c + dt * L
    part = np.abs(dt * L / np.spacing(np.abs(c))) % 1
    clear = big & (np.abs(part - 0.5) > 0.05)  # not a matter of the last rounding
    assert clear.sum() > big.sum() // 2 and (ref != c)[clear].mean() > 0.2
    if scheme == "SSP_RK3":
        assert (np.abs(u - ref) <= 2 * np.spacing(np.abs(ref)))[clear].all()
    else:
        assert np.array_equal(u[clear], ref[clear])
