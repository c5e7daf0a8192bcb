"""The work that users of dgcuda_gb300 have it do, as timed cases.

Every case runs RK-DG time steps through the package's public entry points on
a jittered triangle mesh of the unit square (or the problem's own box): one
problem stepped from a state in device memory, an ensemble stepped as a
batch, or the gradient of a shallow-water run.  A pass hands the solver its
initial state, steps it, and takes the whole result back, so it can be
repeated; the meshes, the initial data and the receivers follow from the seed.

`exact` is the same method written with plain torch operations in 64 bits: an
orthonormal modal basis on each triangle, upwind or local Lax-Friedrichs
fluxes, SSP-RK3 / RK4 / midpoint RK2, the edge-point slope limiter and the
positivity rule, and torch's own autograd for the gradient.
"""
import functools
import math
from fractions import Fraction

import numpy as np
import torch

import dgcuda_gb300 as dg

EQ = {"advection": dg.ADVECTION, "euler": dg.EULER, "shallow_water": dg.SHALLOW_WATER,
      "maxwell": dg.MAXWELL}
NVARS = {"advection": 1, "euler": 4, "shallow_water": 3, "maxwell": 3}
SCHEMES = {"ssp_rk3": dg.SSP_RK3, "rk4": dg.RK4, "rk2": dg.RK2}
STAGES = {"ssp_rk3": 3, "rk4": 4, "rk2": 2}
G = 9.81
GAMMA = 1.4
WALLS = (-1, -1, -1, -1)
OPEN = (-4, -4, -4, -4)
INFLOW = (-3, -3, -3, -3)
PERIODIC = (0, 0, 0, 0)

# what a problem is: equation, box, boundary, mesh jitter, CFL number, package problem name
PROBLEMS = {
    "sine": ("advection", (0.0, 1.0, 0.0, 1.0), PERIODIC, 0.1, 0.3, "adv_sine"),
    "hill": ("advection", (-1.0, 1.0, -1.0, 1.0), INFLOW, 0.1, 0.3, "adv_rotatinghill"),
    "vortex": ("euler", (0.0, 10.0, 0.0, 10.0), PERIODIC, 0.15, 0.2, "euler_vortex"),
    "riemann": ("euler", (0.0, 1.0, 0.0, 1.0), OPEN, 0.1, 0.2, "euler_riemann4"),
    "box": ("euler", (0.0, 1.0, 0.0, 1.0), WALLS, 0.1, 0.3, "none"),
    "hump": ("shallow_water", (0.0, 1.0, 0.0, 1.0), WALLS, 0.1, 0.3, "sw_hump"),
    "wave": ("maxwell", (0.0, 1.0, 0.0, 1.0), WALLS, 0.1, 0.3, "maxwell_plane"),
}


def _case(name, kind, problem, nx, ny, p, steps, scheme="ssp_rk3", limiter=0, bed=0, waves=0.05,
          **more):
    return dict(name=name, kind=kind, problem=problem, nx=nx, ny=ny, p=p, steps=steps,
                scheme=scheme, limiter=limiter, bed=bed, waves=waves, **more)


def listed():
    return [
        # the verification run every new user starts with: scalar advection, 2,048 triangles,
        # lowest order with a slope; a step is a handful of launches on a few blocks
        _case("advection_p1_2k", "step", "sine", 32, 32, 1, 25),
        # a rotating velocity field entering through the boundary, ragged mesh, high order
        _case("advection_hill_p3_35k", "step", "hill", 157, 113, 3, 10),
        # the isentropic vortex accuracy study, 32,768 triangles
        _case("euler_vortex_p3_33k", "step", "vortex", 128, 128, 3, 10),
        # the classical Runge-Kutta loop of the reference program, slip walls, ragged mesh
        _case("euler_box_rk4_p2_60k", "step", "box", 201, 149, 2, 4, scheme="rk4"),
        # shock runs, limiter on: the throughput sweep over the orders.  p = 1 and 3 on the full
        # 2.1 M triangles (p = 3 from the plain Riemann data), p = 2 and 4 on ragged meshes
        # with waves on the background, as a developed flow has
        _case("euler_riemann_p1_2M", "step", "riemann", 1024, 1024, 1, 4, limiter=1),
        _case("euler_riemann_p2_700k", "step", "riemann", 701, 499, 2, 4, limiter=1),
        _case("euler_riemann_p3_2M", "step", "riemann", 1024, 1024, 3, 2, limiter=1, waves=0.0),
        _case("euler_riemann_p4_500k", "step", "riemann", 503, 497, 4, 2, limiter=1),
        # a basin over a sine bed with reflecting walls, 131,072 triangles
        _case("shallow_water_p2_131k", "step", "hump", 256, 256, 2, 10, bed=1),
        # an ensemble of uneven problems stepped together (parameter studies)
        _case("shallow_water_ensemble", "batch", "hump", 0, 0, 0, 4, members=24, tri_min=1000,
              tri_max=200000),
        # gradient of a receiver misfit with respect to the initial state and the bed
        _case("shallow_water_gradient_p2", "gradient", "hump", 150, 150, 2, 10, bed=1, every=5,
              receivers=64),
        # a cavity with conducting walls, ragged mesh, high order
        _case("maxwell_p3_126k", "step", "wave", 299, 211, 3, 5),
    ]


def draw(rng):
    kind = rng.choice(["step"] * 8 + ["batch", "gradient"])
    if kind == "batch":
        return {k: v for k, v in _case(
            "", "batch", "hump", 0, 0, 0, rng.randint(2, 4), members=rng.randint(5, 24),
            tri_min=rng.randint(300, 2000), tri_max=rng.randint(20000, 200000)).items()
            if k != "name"}
    problem = rng.choice(["sine", "hill", "vortex", "riemann", "riemann", "box", "hump", "wave"])
    p = rng.randint(1, 4)
    if kind == "gradient":
        problem, p = "hump", rng.randint(1, 3)
    top = {"gradient": 60000}.get(kind, 1500000 // (p + 1))
    tri = math.exp(rng.uniform(math.log(500), math.log(top)))
    shape = math.exp(rng.uniform(-0.5, 0.5))
    nx = max(4, round(math.sqrt(tri / 2) * shape))
    ny = max(4, round(tri / 2 / nx))
    steps = rng.randint(2, 4) if tri > 100000 else rng.randint(4, 12)
    more = {}
    scheme = "ssp_rk3"
    limiter = 1 if problem == "riemann" else 0
    if kind == "gradient":
        more = dict(every=rng.randint(1, 3), receivers=rng.randint(1, 80))
    elif problem in ("vortex", "box") and rng.random() < 0.4:
        scheme = rng.choice(["rk4", "rk2"])
    bed = int(problem == "hump" and rng.random() < 0.5)
    c = _case("", kind, problem, nx, ny, p, steps, scheme, limiter, bed,
              round(rng.uniform(0.01, 0.08), 3), **more)
    del c["name"]
    return c


def _sizes(p):
    return (p + 1) * (p + 2) // 2, {1: 3, 2: 6, 3: 12, 4: 16}[p], p + 1


def _step_work(K, N, p, steps, scheme, bed=False):
    """Bytes and flops of `steps` steps: each stage reads its input and writes its output, the
    combinations of the later stages read u^n too; 56 bytes of geometry per element and stage."""
    npm, nq, n1 = _sizes(p)
    s = STAGES[scheme]
    streams = 3 * s - 1
    by = K * (8 * N * npm * streams + 56 * s + (8 * npm * s if bed else 0)) * steps
    vol = nq * N * npm * 2 + nq * N * 8 + nq * N * (npm - 1) * 4
    fl = K * (vol + 3 * n1 * N * npm * 4 + N * npm * 6) * s * steps
    return by, fl


def work(case):
    if case["kind"] == "batch":
        by = fl = 0
        for m in _members(case, 1):
            b, f = _step_work(2 * m["side"] ** 2, 3, m["p"], case["steps"], "ssp_rk3", m["bed"])
            by, fl = by + b, fl + f
        return {"bytes": by, "flops": fl}
    K, N = 2 * case["nx"] * case["ny"], NVARS[PROBLEMS[case["problem"]][0]]
    by, fl = _step_work(K, N, case["p"], case["steps"], case["scheme"], case["bed"])
    if case["kind"] == "gradient":  # forward, and the transposed operator once per stage
        by, fl = 3 * by, 3 * fl
    return {"bytes": by, "flops": fl}


# ---------------------------------------------------------------------------
# inputs, from the seed alone
# ---------------------------------------------------------------------------
def _members(case, seed):
    rng = np.random.default_rng(seed)
    sizes = np.random.default_rng(77)  # the ensemble's sizes and orders: the same for every seed
    out = []
    for _ in range(case["members"]):
        tri = math.exp(sizes.uniform(math.log(case["tri_min"]), math.log(case["tri_max"])))
        out.append(dict(side=max(4, round(math.sqrt(tri / 2))), p=int(sizes.integers(1, 4)),
                        bed=int(sizes.uniform() < 0.5), seed=int(rng.integers(1, 2 ** 31))))
    return out


@functools.lru_cache(maxsize=6)
def _mesh(problem, nx, ny, seed):
    _, box, bc, jitter, _, _ = PROBLEMS[problem]
    return dg.Mesh.square(nx, ny, box=box, jitter=jitter, seed=seed, bc=bc)


def _device():
    return torch.device("cuda") if torch.cuda.is_available() else torch.device("cpu")


def _points(V, r, s):
    """Coordinates of reference points (r, s) in every element, [points, K]."""
    r, s = (torch.as_tensor(x, dtype=torch.float64, device=V.device)[:, None] for x in (r, s))
    return (V[0] + (V[2] - V[0]) * r + (V[4] - V[0]) * s,
            V[1] + (V[3] - V[1]) * r + (V[5] - V[1]) * s)


def _ripples(rng, box):
    """A smooth function of position with values in about [-1, 1]."""
    lx, ly = box[1] - box[0], box[3] - box[2]
    terms = [(rng.uniform(0.1, 0.35), int(rng.integers(1, 5)), int(rng.integers(1, 5)),
              rng.uniform(0, 2 * math.pi)) for _ in range(4)]

    def f(x, y):
        return sum(a * torch.sin(2 * math.pi * (k * (x - box[0]) / lx + m * (y - box[2]) / ly) + ph)
                   for a, k, m, ph in terms)
    return f


def _rotated_hill(x, y, t):
    c, s = math.cos(2 * math.pi * t), math.sin(2 * math.pi * t)
    dx, dy = x * c + y * s - 0.2, -x * s + y * c
    return 5.0 * torch.exp(-(dx * dx + dy * dy) / (2 * 0.15 ** 2))


def _vortex_prm(seed):
    return (float(np.random.default_rng(seed + 1000).uniform(4.0, 5.5)), 5.0, 5.0, 1.0, 1.0, 10.0)


def _hump(seed):
    rng = np.random.default_rng(seed + 2000)
    return (1.0, rng.uniform(0.05, 0.2), rng.uniform(0.05, 0.15), rng.uniform(0.2, 0.8),
            rng.uniform(0.2, 0.8))


def _initial(problem, waves, seed, x, y):
    """Conserved variables at the points, a list of [points, K]."""
    rng = np.random.default_rng(seed)
    f = _ripples(rng, PROBLEMS[problem][1])
    if problem == "sine":
        return [torch.sin(2 * math.pi * x) * torch.sin(2 * math.pi * y) + waves * f(x, y)]
    if problem == "hill":
        return [_rotated_hill(x, y, 0.0) * (1 + waves * f(x, y))]
    if problem == "wave":
        g, h = _ripples(rng, PROBLEMS[problem][1]), _ripples(rng, PROBLEMS[problem][1])
        return [f(x, y), g(x, y), h(x, y)]
    if problem == "hump":
        h0, A, sig, x0, y0 = _hump(seed)
        h = h0 + A * torch.exp(-((x - x0) ** 2 + (y - y0) ** 2) / sig ** 2)
        return [h, torch.zeros_like(h), torch.zeros_like(h)]
    if problem == "vortex":
        beta, x0, y0, ui, vi, _ = _vortex_prm(seed)
        dx, dy = x - x0, y - y0
        e = torch.exp(0.5 * (1 - dx * dx - dy * dy))
        u, v = ui - beta / (2 * math.pi) * e * dy, vi + beta / (2 * math.pi) * e * dx
        T = 1 - (GAMMA - 1) * beta ** 2 / (8 * GAMMA * math.pi ** 2) * e * e
        rho = T ** (1 / (GAMMA - 1))
        pr = rho ** GAMMA
    elif problem == "box":
        g = _ripples(rng, PROBLEMS[problem][1])
        rho, u, v, pr = 1 + waves * f(x, y), 0.3 * g(x, y), 0.2 * f(x, y), 1 + waves * g(x, y)
    else:  # four-quadrant Riemann data; the waves scale the conserved variables
        left, low = x < 0.5, y < 0.5
        ne, nw, sw, se = ((1.5, 0., 0., 1.5), (0.5323, 1.206, 0., 0.3), (0.138, 1.206, 1.206, 0.029),
                          (0.5323, 0., 1.206, 0.3))
        rho, u, v, pr = (torch.where(left, torch.where(low, c, b), torch.where(low, d, a))
                         for a, b, c, d in ([torch.tensor(q, dtype=torch.float64, device=x.device)
                                             for q in quad] for quad in zip(ne, nw, sw, se)))
    U = [rho, rho * u, rho * v, 0.5 * rho * (u * u + v * v) + pr / (GAMMA - 1)]
    if problem == "riemann" and waves:
        scale = 1 + waves * f(x, y)
        U = [a * scale for a in U]
    return U


def _bed(x, y):
    return 0.1 * torch.sin(2 * math.pi * x) * torch.sin(2 * math.pi * y)


def _project(values, tab):
    """Modes [i][K] of values [points, K] at the area points."""
    wB = torch.as_tensor(tab["w"][:, None] * tab["B"], device=values.device)
    return wB.T @ values


def _state(problem, waves, seed, V, p):
    tab = _tables(p)
    x, y = _points(V, tab["r"], tab["s"])
    return torch.stack([_project(u, tab) for u in _initial(problem, waves, seed, x, y)])


def _vertices(mesh):
    return torch.as_tensor(mesh.arrays()[0], device=_device())


def _receivers(n, seed):
    rng = np.random.default_rng(seed + 3000)
    return rng.uniform(0.05, 0.95, n), rng.uniform(0.05, 0.95, n)


def _sbar(case, seed):
    rng = np.random.default_rng(seed + 4000)
    return rng.standard_normal((case["steps"] // case["every"], case["receivers"]))


def _gradient_dt(case):
    # a fixed step, 0.05 of the cell over the largest wave speed met (below 4)
    return 0.05 / max(case["nx"], case["ny"]) / (2 * case["p"] + 1)


# ---------------------------------------------------------------------------
# what a user's program holds, and one pass
# ---------------------------------------------------------------------------
def _solver(problem, mesh, p, seed, waves, limiter, bed):
    eq, _, _, _, cfl, name = PROBLEMS[problem]
    prm = {"vortex": _vortex_prm, "hump": _hump}.get(problem, lambda _: ())(seed)
    s = dg.Solver(mesh, EQ[eq], p, problem=name, limiter=limiter, cfl=cfl, gravity=G, prm=prm)
    V = _vertices(mesh)
    c0 = _state(problem, waves, seed, V, p).contiguous()
    if bed:
        tab = _tables(p)
        s.set_bathymetry(_project(_bed(*_points(V, tab["r"], tab["s"])), tab).cpu().numpy())
    return s, c0


def prepare(case, seed):
    if case["kind"] == "batch":
        got = []
        for m in _members(case, seed):
            mesh = _mesh("hump", m["side"], m["side"], m["seed"])
            got.append(_solver("hump", mesh, m["p"], m["seed"], 0.0, 0, m["bed"]))
        solvers, c0 = [s for s, _ in got], [c for _, c in got]
        return dict(case=case, solvers=solvers, batch=dg.Batch(solvers), c0=c0,
                    out=[torch.empty_like(c) for c in c0])
    mesh = _mesh(case["problem"], case["nx"], case["ny"], seed)
    s, c0 = _solver(case["problem"], mesh, case["p"], seed, case["waves"], case["limiter"],
                    case["bed"])
    st = dict(case=case, solver=s, c0=c0, out=torch.empty_like(c0))
    if case["kind"] == "gradient":
        st["adjoint"] = dg.Adjoint(s, *_receivers(case["receivers"], seed))
        st["sbar"] = _sbar(case, seed)
        st["dt"] = _gradient_dt(case)
    return st


def _put(solver, c):
    """dg_set_state_device (dg.h): the state from device memory."""
    if dg.load_library().dg_set_state_device(solver._h, c.data_ptr()):
        raise RuntimeError(dg.load_library().dg_last_error().decode())


def _get(solver, out):
    """dg_get_state_device (dg.h): the state into device memory."""
    if dg.load_library().dg_get_state_device(solver._h, out.data_ptr()):
        raise RuntimeError(dg.load_library().dg_last_error().decode())
    return out


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        for s, c in zip(state["solvers"], state["c0"]):
            _put(s, c)
        t = state["batch"].step(case["steps"])
        return {"t": t, "u": [_get(s, o) for s, o in zip(state["solvers"], state["out"])]}
    s = state["solver"]
    _put(s, state["c0"])
    if case["kind"] == "gradient":
        samples = state["adjoint"].forward(case["steps"], state["dt"], case["every"])
        gu, gb = state["adjoint"].backward(state["sbar"])
        return {"samples": samples, "grad_u0": gu, "grad_b": gb}
    t = s.step(case["steps"], SCHEMES[case["scheme"]], 0.0)
    return {"t": t, "u": _get(s, state["out"])}


# ---------------------------------------------------------------------------
# the method in plain torch, 64 bits
# ---------------------------------------------------------------------------
def _orbit3(a, w):
    a, w = Fraction(a), Fraction(w)
    return [(1 - 2 * a, a, w), (a, 1 - 2 * a, w), (a, a, w)]


def _orbit6(p, order, w):
    p = [Fraction(v) for v in p]
    return [(p[i], p[j], Fraction(w)) for i, j in order]


def _area_rule(p):
    """Dunavant's symmetric rule of degree 2 p (15 published digits), weights summing to 1."""
    if p == 1:
        return [(Fraction(1, 6), Fraction(1, 6), Fraction(1, 3)),
                (Fraction(2, 3), Fraction(1, 6), Fraction(1, 3)),
                (Fraction(1, 6), Fraction(2, 3), Fraction(1, 3))]
    if p == 2:
        return (_orbit3("0.091576213509771", "0.109951743655322") +
                _orbit3("0.445948490915965", "0.223381589678011"))
    if p == 3:
        return (_orbit3("0.063089014491502", "0.050844906370207") +
                _orbit3("0.249286745170910", "0.116786275726379") +
                _orbit6(("0.636502499121399", "0.310352451033784", "0.053145049844817"),
                        [(0, 1), (1, 0), (0, 2), (1, 2), (2, 1), (2, 0)], "0.082851075618374"))
    return ([(Fraction(1, 3), Fraction(1, 3), Fraction("0.144315607677787"))] +
            _orbit3("0.459292588292723", "0.095091634267285") +
            _orbit3("0.170569307751760", "0.103217370534718") +
            _orbit3("0.050547228317031", "0.032458497623198") +
            _orbit6(("0.008394777409958", "0.728492392955404", "0.263112829634638"),
                    [(0, 1), (1, 0), (2, 0), (0, 2), (2, 1), (1, 2)], "0.027230314174435"))


@functools.lru_cache(maxsize=None)
def _basis(p):
    """Orthonormal polynomials on the unit triangle, as [({(a, b): coefficient}, norm^2)]:
    Gram-Schmidt over 1, r, s, r^2, r s, s^2, ... in rational arithmetic."""
    monomials = [(d - j, j) for d in range(p + 1) for j in range(d + 1)]

    def inner(f, g):
        return sum(c * e * Fraction(math.factorial(a + k) * math.factorial(b + m),
                                    math.factorial(a + b + k + m + 2))
                   for (a, b), c in f.items() for (k, m), e in g.items())

    done = []
    for mono in monomials:
        f = {mono: Fraction(1)}
        for g, nn in done:
            c = inner({mono: Fraction(1)}, g) / nn
            for k, e in g.items():
                f[k] = f.get(k, Fraction(0)) - c * e
        done.append((f, inner(f, f)))
    return done


def _value(f, nn, r, s):
    return float(sum(c * r ** a * s ** b for (a, b), c in f.items())) / math.sqrt(nn)


def _slope(f, nn, r, s, k):
    v = sum(c * (a, b)[k] * r ** (a - (k == 0)) * s ** (b - (k == 1))
            for (a, b), c in f.items() if (a, b)[k])
    return float(v) / math.sqrt(nn)


@functools.lru_cache(maxsize=None)
def _tables(p):
    rule, basis = _area_rule(p), _basis(p)
    t1, w1 = np.polynomial.legendre.leggauss(p + 1)
    w = np.array([float(q[2]) / 2 for q in rule])

    def at(points):
        return np.array([[_value(f, nn, r, s) for f, nn in basis] for r, s in points])

    half = [Fraction(float(t)) / 2 + Fraction(1, 2) for t in t1]
    edges = np.stack([at([(h, Fraction(0)) for h in half]), at([(1 - h, h) for h in half]),
                      at([(Fraction(0), 1 - h) for h in half])])
    area = [(q[0], q[1]) for q in rule]
    return dict(r=np.array([float(a) for a, _ in area]), s=np.array([float(b) for _, b in area]),
                w=w, B=at(area), E=edges, t1=t1, w1=w1,
                GR=w[:, None] * np.array([[_slope(f, nn, r, s, 0) for f, nn in basis]
                                          for r, s in area]),
                GS=w[:, None] * np.array([[_slope(f, nn, r, s, 1) for f, nn in basis]
                                          for r, s in area]))


class _Exact:
    """One problem: its mesh as torch tensors and the DG operator on states [var][mode][K]."""

    def __init__(self, problem, mesh, p, limiter=0, bed=None):
        self.problem, self.p, self.limiter = problem, p, limiter
        self.eq, self.box, _, _, self.cfl, _ = PROBLEMS[problem]
        dev = _device()
        V, es, _, se = mesh.arrays()
        self.V = torch.as_tensor(V, device=dev)
        self.es = torch.as_tensor(es.astype(np.int64), device=dev)
        left, right, lf, rf = torch.as_tensor(se.astype(np.int64), device=dev)
        self.left, self.lf, self.rf, self.right = left, lf, rf, right
        self.tab = {k: torch.as_tensor(v, device=dev) for k, v in _tables(p).items()}
        x1, y1, x2, y2, x3, y3 = self.V
        self.xr, self.yr, self.xs, self.ys = x2 - x1, y2 - y1, x3 - x1, y3 - y1
        self.J = self.xr * self.ys - self.xs * self.yr
        a, b, c = (torch.hypot(x1 - x2, y1 - y2), torch.hypot(x2 - x3, y2 - y3),
                   torch.hypot(x1 - x3, y1 - y3))
        k = 0.5 * (a + b + c)
        self.dmin = float((2 * torch.sqrt(k * (k - a) * (k - b) * (k - c)) / k).min())
        # the left element's face runs from vertex lf to lf + 1, counter-clockwise
        vb = (lf + 1) % 3
        self.ax, self.ay = self.V[2 * lf, left], self.V[2 * lf + 1, left]
        self.bx, self.by = self.V[2 * vb, left], self.V[2 * vb + 1, left]
        dx, dy = self.bx - self.ax, self.by - self.ay
        self.len = torch.hypot(dx, dy)
        self.nx, self.ny = dy / self.len, -dx / self.len
        own = torch.arange(self.V.shape[1], device=dev)
        self.is_left = torch.stack([(left[self.es[f]] == own) & (lf[self.es[f]] == f)
                                    for f in range(3)])
        other = torch.stack([torch.where(self.is_left[f], right[self.es[f]], left[self.es[f]])
                             for f in range(3)])
        self.nbr = torch.where(other >= 0, other, own)
        self.ends = right < 0
        self.bed = None if bed is None else torch.as_tensor(bed, device=dev)

    # ---- the equations
    def velocity(self, x, y):
        if self.problem == "hill":
            return -2 * math.pi * y, 2 * math.pi * x
        return torch.full_like(x, 1.0), torch.full_like(x, 0.5)

    def flux(self, U, x, y):
        if self.eq == "advection":
            vx, vy = self.velocity(x, y)
            return [vx * U[0]], [vy * U[0]]
        if self.eq == "maxwell":
            z = torch.zeros_like(U[0])
            return [z, U[2], U[1]], [-U[2], z, -U[0]]
        u, v = U[1] / U[0], U[2] / U[0]
        if self.eq == "shallow_water":
            hp = 0.5 * G * U[0] * U[0]
            return [U[1], U[1] * u + hp, U[1] * v], [U[2], U[2] * u, U[2] * v + hp]
        pr = (GAMMA - 1) * (U[3] - 0.5 * (U[1] * u + U[2] * v))
        return ([U[1], U[1] * u + pr, U[1] * v, (U[3] + pr) * u],
                [U[2], U[2] * u, U[2] * v + pr, (U[3] + pr) * v])

    def speed(self, U, nx, ny):
        """|u . n| + c at a trace."""
        if self.eq == "maxwell":
            return torch.ones_like(U[0])
        un = torch.abs((U[1] * nx + U[2] * ny) / U[0])
        if self.eq == "shallow_water":
            return un + torch.sqrt(G * U[0])
        pr = (GAMMA - 1) * (U[3] - 0.5 * (U[1] * U[1] + U[2] * U[2]) / U[0])
        return un + torch.sqrt(GAMMA * pr / U[0])

    def largest(self, c):
        B0 = self.tab["B"][0, 0]
        if self.eq == "maxwell":
            return 1.0
        if self.problem == "hill":
            k = len(self.tab["r"]) // 2
            x, y = _points(self.V, self.tab["r"][k:k + 1], self.tab["s"][k:k + 1])
            return float(torch.hypot(*self.velocity(x, y)).max())
        if self.problem == "sine":
            return math.hypot(1.0, 0.5)
        U = [c[n, 0] * B0 for n in range(c.shape[0])]
        un = torch.hypot(U[1], U[2]) / U[0]
        if self.eq == "shallow_water":
            return float((un + torch.sqrt(G * U[0])).max())
        pr = (GAMMA - 1) * (U[3] - 0.5 * (U[1] ** 2 + U[2] ** 2) / U[0])
        return float((un + torch.sqrt(GAMMA * pr / U[0])).max())

    def physical(self, U):
        """Per element: every point of U, a list of [..., K], is physical."""
        if self.eq in ("advection", "maxwell"):
            return None
        ok = U[0] >= 0
        if self.eq == "euler":
            ok = ok & (2 * U[0] * U[3] >= U[1] * U[1] + U[2] * U[2])
        return ok.flatten(0, -2).all(dim=0)

    # ---- the operator
    def traces(self, c):
        """[var][3][n1][K]"""
        E = self.tab["E"]
        return (E.reshape(-1, E.shape[2]) @ c).reshape(c.shape[0], 3, E.shape[1], c.shape[2])

    def ghost(self, UL, t, nx, ny, x, y):
        code = int(self.right[self.ends][0])
        if code == -4:
            return UL
        if code == -3:
            return [_rotated_hill(x, y, t)]
        if self.eq == "maxwell":
            dot = UL[0] * nx + UL[1] * ny
            return [2 * dot * nx - UL[0], 2 * dot * ny - UL[1], UL[2]]
        dot = UL[1] * nx + UL[2] * ny
        return [UL[0], UL[1] - 2 * dot * nx, UL[2] - 2 * dot * ny] + list(UL[3:])

    def side_fluxes(self, T, t):
        """[var][n1][S], times len / 2 and the edge weights"""
        out = []
        for j in range(self.p + 1):
            h = 0.5 + 0.5 * self.tab["t1"][j]
            x, y = self.ax + h * (self.bx - self.ax), self.ay + h * (self.by - self.ay)
            UL = T[:, self.lf, j, self.left]
            UR = T[:, self.rf.clamp(min=0), self.p - j, self.right.clamp(min=0)]
            if bool(self.ends.any()):
                e = self.ends
                g = self.ghost(list(UL[:, e]), t, self.nx[e], self.ny[e], x[e], y[e])
                UR = UR.masked_scatter(e.expand_as(UR), torch.stack(g))
            UL, UR = list(UL), list(UR)
            if self.eq == "advection":
                vx, vy = self.velocity(x, y)
                an = self.nx * vx + self.ny * vy
                F = [torch.where(an > 0, an * UL[0], an * UR[0])]
            else:
                fl, gl = self.flux(UL, x, y)
                fr, gr = self.flux(UR, x, y)
                lam = torch.maximum(self.speed(UL, self.nx, self.ny),
                                    self.speed(UR, self.nx, self.ny))
                F = [0.5 * ((a + b) * self.nx + (k + m) * self.ny + lam * (l - r))
                     for a, b, k, m, l, r in zip(fl, fr, gl, gr, UL, UR)]
            out.append(torch.stack(F) * (self.len / 2 * self.tab["w1"][j]))
        return torch.stack(out, dim=1)

    def rhs(self, c, t, T=None):
        """(du/dt, c with the elements whose area values are not physical set to their means)"""
        tab = self.tab
        T = self.traces(c) if T is None else T
        Fs = self.side_fluxes(T, t)
        U = tab["B"] @ c
        ok = self.physical(list(U))
        if ok is not None and not bool(ok.all()):
            keep = torch.zeros_like(c)
            keep[:, 0] = 1.0
            c = torch.where(ok, c, c * keep)
            U = tab["B"] @ c
        x, y = _points(self.V, tab["r"], tab["s"])
        fx, fy = (torch.stack(f) for f in self.flux(list(U), x, y))
        acc = (tab["GR"].T @ (fx * self.ys - fy * self.xs) +
               tab["GS"].T @ (fy * self.xr - fx * self.yr))
        if self.bed is not None:
            br, bs = tab["GR"] @ self.bed, tab["GS"] @ self.bed
            sx = -G * U[0] * (self.ys * br - self.yr * bs)
            sy = -G * U[0] * (self.xr * bs - self.xs * br)
            acc = acc + torch.stack([torch.zeros_like(acc[0]), tab["B"].T @ sx, tab["B"].T @ sy])
        for f in range(3):
            F = Fs[:, :, self.es[f]]
            F = torch.where(self.is_left[f], -F, F.flip(1))
            acc = acc + tab["E"][f].T @ F
        return acc / self.J, c

    def limit(self, c):
        if not self.limiter:
            return c
        phi0 = self.tab["B"][0, 0]
        mean = c[:, 0] * phi0
        around = torch.stack([mean] + [mean[:, self.nbr[f]] for f in range(3)])
        low, high = mean - around.amin(dim=0), around.amax(dim=0) - mean
        d = self.traces(c) - mean[:, None, None]
        up, down = d.amax(dim=(1, 2)).clamp(min=0), (-d).amax(dim=(1, 2)).clamp(min=0)
        one = torch.ones_like(mean)
        alpha = torch.minimum(torch.where(up > low, low / torch.where(up > 0, up, one), one),
                              torch.where(down > high, high / torch.where(down > 0, down, one), one))
        out = c.clone()
        cut = alpha < 1
        out[:, 1] = c[:, 1] * alpha
        out[:, 2] = c[:, 2] * alpha
        if c.shape[1] > 3:
            out[:, 3:] = torch.where(cut[:, None], torch.zeros_like(c[:, 3:]), c[:, 3:])
        return out

    def settle(self, c):
        """Elements with a non-physical edge value set to their means; (c, traces)"""
        T = self.traces(c)
        ok = self.physical(list(T))
        if ok is not None and not bool(ok.all()):
            keep = torch.zeros_like(c)
            keep[:, 0] = 1.0
            c = torch.where(ok, c, c * keep)
            T = self.traces(c)
        return c, T

    def ssp_rk3(self, u, t, dt):
        """u: limited and settled"""
        L, u = self.rhs(u, t)
        w, T = self.settle(self.limit(u + dt * L))
        L, w = self.rhs(w, t + dt, T)
        w, T = self.settle(self.limit(0.75 * u + 0.25 * w + 0.25 * dt * L))
        L, w = self.rhs(w, t + 0.5 * dt, T)
        return self.settle(self.limit(u / 3 + 2 / 3 * w + 2 / 3 * dt * L))[0]

    def dt(self, c):
        return self.cfl * self.dmin / self.largest(c) / (2 * self.p + 1)

    def run(self, u, steps, scheme):
        t = 0.0
        u = self.limit(u)
        if scheme == "ssp_rk3":
            u = self.settle(u)[0]
        for _ in range(steps):
            dt = self.dt(u)
            if scheme == "ssp_rk3":
                u = self.ssp_rk3(u, t, dt)
                t += dt
                continue
            t += dt

            def k(v, at):
                v, T = self.settle(v)
                return self.limit(dt * self.rhs(v, at, T)[0])
            k1 = k(u, t)
            if scheme == "rk2":
                u = self.limit(u + k(u + 0.5 * k1, t + 0.5 * dt))
                continue
            k2 = k(u + 0.5 * k1, t + 0.5 * dt)
            k3 = k(u + 0.5 * k2, t + 0.5 * dt)
            k4 = k(u + k3, t + dt)
            u = self.limit(u + k1 / 6 + k2 / 3 + k3 / 3 + k4 / 6)
        return u, t


def _exact_problem(problem, mesh, p, seed, waves, limiter, bed):
    V = _vertices(mesh)
    b = None
    if bed:
        tab = _tables(p)
        b = _project(_bed(*_points(V, tab["r"], tab["s"])), tab)
    return _Exact(problem, mesh, p, limiter, b), _state(problem, waves, seed, V, p)


def _sampler(E, case, seed):
    """(element, basis values) of each receiver"""
    rx, ry = (torch.as_tensor(v, device=E.V.device)[:, None] for v in
              _receivers(case["receivers"], seed))
    dx, dy = rx - E.V[0], ry - E.V[1]
    r, s = (E.ys * dx - E.xs * dy) / E.J, (E.xr * dy - E.yr * dx) / E.J
    inside = torch.minimum(torch.minimum(r, s), 1 - r - s)
    el = inside.argmax(dim=1)
    at = torch.arange(len(el), device=el.device)
    phi = [[_value(f, nn, float(a), float(b)) for f, nn in _basis(case["p"])]
           for a, b in zip(r[at, el].tolist(), s[at, el].tolist())]
    return el, torch.tensor(phi, dtype=torch.float64, device=el.device)


def exact(case, seed):
    if case["kind"] == "batch":
        ts, us = [], []
        for m in _members(case, seed):
            mesh = _mesh("hump", m["side"], m["side"], m["seed"])
            E, c0 = _exact_problem("hump", mesh, m["p"], m["seed"], 0.0, 0, m["bed"])
            u, t = E.run(c0, case["steps"], "ssp_rk3")
            ts.append(t)
            us.append(u)
        return {"t": np.array(ts), "u": us}
    mesh = _mesh(case["problem"], case["nx"], case["ny"], seed)
    E, c0 = _exact_problem(case["problem"], mesh, case["p"], seed, case["waves"],
                           case["limiter"], case["bed"])
    if case["kind"] == "step":
        u, t = E.run(c0, case["steps"], case["scheme"])
        return {"t": t, "u": u}
    dt, every = _gradient_dt(case), case["every"]
    el, phi = _sampler(E, case, seed)
    if E.bed is None:
        E.bed = torch.zeros_like(c0[0])
    u0, b = c0.clone().requires_grad_(True), E.bed.clone().requires_grad_(True)
    E.bed = b
    u, samples = u0, []
    for n in range(case["steps"]):
        u = E.ssp_rk3(u, n * dt, dt)
        if (n + 1) % every == 0:
            samples.append((u[0][:, el].T * phi).sum(dim=1))
    samples = torch.stack(samples)
    weights = torch.as_tensor(_sbar(case, seed), device=samples.device)
    gu, gb = torch.autograd.grad((samples * weights).sum(), (u0, b))
    return {"samples": samples.detach(), "grad_u0": gu, "grad_b": gb}
