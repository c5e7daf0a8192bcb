"""The two-limb tables of the element stage's fixed-point contractions,
checked on the CPU with Python integers: they reproduce the basis tables,
no sum of products can leave 64 bits, and a contraction done the kernel's way
is no farther from the exact dot product than FP64 multiply-adds are."""
from fractions import Fraction

import numpy as np
import pytest

LOW = 28


def unit(M):
    """2^(M - 1078)"""
    return Fraction(2) ** (M - 1078)


def limbs(T):
    h = (T + (1 << (LOW - 1))) >> LOW
    return h, T - (h << LOW)


def sums(p, t):
    """Every set of table entries that meets in one sum, with the unit's exponent."""
    nm = (p + 1) * (p + 2) // 2
    for row in t["B"]:
        yield row, t["eB"]
    for row in t["E"]:
        yield row, t["eE"]
    for i in range(nm):
        yield np.concatenate([t["S"][:, i], t["G"][:, 0, i], t["G"][:, 1, i], t["Q"][:, i]]), t["eP"]
    for row in t["G"].reshape(-1, nm):
        yield row, t["eP"]


def entries(*parts):
    """The entries of tables that are not zeros or their roundings, sorted."""
    a = np.sort(np.concatenate([np.ravel(x) for x in parts]))
    return a[np.abs(a) > 1e-14]


@pytest.mark.parametrize("p", [1, 2, 3, 4])
def test_limbs_reproduce_the_tables_and_no_sum_leaves_64_bits(dglib, p):
    t = dglib.fx_table_image(p)
    dense = dglib.oz_table_image(p)[2]  # the FP64 tables, padded with zeros
    val = {k: np.vectorize(lambda v, M=M: float(int(v) * unit(M)))(t[k])
           for k, M in (("B", t["eB"]), ("E", t["eE"]), ("G", t["eP"]), ("S", t["eP"]),
                        ("Q", t["eP"]))}
    # within half a unit, and half an ulp of the comparison's own rounding
    for a, b, M in ((entries(val["B"]), entries(dense[0]), t["eB"]),
                    (entries(val["E"]), entries(dense[4]), t["eE"]),
                    (entries(val["S"], val["G"]), entries(dense[1:4]), t["eP"])):
        assert a.shape == b.shape
        assert np.abs(a - b).max() <= float(unit(M)) / 2 + 2.0 ** -53 * np.abs(b).max()
    assert np.abs(val["Q"] - val["B"]).max() <= float(unit(max(t["eB"], t["eP"])))
    xh, xl = 2 ** 29, 2 ** 27  # the largest limbs of the 57-bit inputs
    for T, _ in sums(p, t):
        th, tl = limbs(T)
        assert np.abs(th).max() < 2 ** 31
        H = sum(xh * abs(int(v)) for v in th)
        M = sum(xh * abs(int(v)) for v in tl) + sum(xl * abs(int(v)) for v in th)
        assert H < 2 ** 62.5 and M + 2 ** (LOW - 1) < 2 ** 63
        assert H + (M >> LOW) < 2 ** 63 - 1


def fixed_dot(x, T, M):
    """The kernel's contraction: limbs of the row's inputs, three products each."""
    ex = int(np.frexp(np.abs(x).max())[1]) - 1
    H, Mm = 0, 1 << (LOW - 1)
    for v, t in zip(x, T):
        a = int(abs(Fraction(v)) * Fraction(2) ** (56 - ex))
        s = 1 if v >= 0 else -1
        h = (a + 2 ** (LOW - 1)) >> LOW
        h, l = s * h, s * (a - (h << LOW))
        th, tl = limbs(int(t))
        H += h * th
        Mm += h * tl + l * th
    return float((H + (Mm >> LOW)) * Fraction(2) ** (2 * LOW + ex - 56) * unit(M))


def fp64_dot(x, t):
    a = 0.0
    for v, w in zip(x, t):
        a = float(Fraction(a) + Fraction(v) * Fraction(w))
    return a


@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("what", ["values", "traces", "projection"])
def test_contractions_are_no_farther_from_exact_than_fp64(dglib, p, what):
    t = dglib.fx_table_image(p)
    nm = (p + 1) * (p + 2) // 2
    rng = np.random.default_rng(p)
    # modes that decay from a mean of 1 to 2
    deg = np.array([d for d in range(p + 1) for _ in range(d + 1)])
    rows = rng.uniform(-1, 1, (24, nm)) * 0.3 ** deg
    rows[:, 0] = rng.uniform(1, 2, 24)
    if what == "values":
        cols, M = list(t["B"]), t["eB"]
    elif what == "traces":
        cols, M = list(t["E"]), t["eE"]
    else:  # their advection on the reference triangle: fluxes at the edge and area points
        U = rows @ np.array([[float(int(v) * unit(t["eB"])) for v in T] for T in t["B"]]).T
        Ue = rows @ np.array([[float(int(v) * unit(t["eE"])) for v in T] for T in t["E"]]).T
        v = rng.uniform(-1, 1, (24, 2))
        w = 0.5 * np.polynomial.legendre.leggauss(p + 1)[1]
        n = np.repeat([[0, -1], [1, 1], [-1, 0]], p + 1, axis=0)
        rows = np.concatenate([-np.tile(w, 3) * (v @ n.T) * Ue, v[:, :1] * U, v[:, 1:] * U], axis=1)
        T = np.concatenate([t["S"], t["G"][:, 0], t["G"][:, 1]])
        cols, M = [T[:, i] for i in range(nm)], t["eP"]
    fx = fp = 0.0
    for x in rows:
        for T in cols:
            tab = [int(v) * unit(M) for v in T]
            exact = sum((Fraction(v) * w for v, w in zip(x, tab)), Fraction(0))
            # FP64 against its own rounded table entries: its additions alone
            t64 = [float(w) for w in tab]
            exact64 = sum((Fraction(v) * Fraction(w) for v, w in zip(x, t64)), Fraction(0))
            fx += float(Fraction(fixed_dot(x, T, M)) - exact) ** 2
            fp += float(Fraction(fp64_dot(x, t64)) - exact64) ** 2
    print(what, p, (fx / len(rows) / len(cols)) ** 0.5, (fp / len(rows) / len(cols)) ** 0.5)
    assert fx <= fp
