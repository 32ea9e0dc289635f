"""The functions of the FP64 pair kernels (1/sqrt, 1/x, exp(-x^2) and erfcx by
their own Newton steps and polynomials) pair by pair, against 50-digit decimal
arithmetic: isolated pairs on a lattice, each with a distance of its own whose
square FP64 holds exactly, over everything the fast form takes (alpha r from 0
to 6, both ends, r from 2e-3 A).

Tolerances, first-order worst cases in units of u = 2^-53 (an operation's
rounding is at most 1 u):
  1/sqrt 1.5; sqrt and alpha r 2;
  erfcx: argument 2, (x - 3) / (x + 3) 4 (times at most 1.2 in the result),
    Horner scheme 3.2, the last product 3; at most 11 together;
  exp(-x^2) from the two-part product 3.2;
  an energy C q q exp erfcx / r: 11 + 3.2 + 1.5 and three products, 19;
  r dE/dr: the energy or the second term (less), and the sum, 20;
  a force: that, 1/r^2 within 1, two products, 23;
  a sum over blocks: three additions more, 22 and 23.
"""
import decimal
import math
from decimal import Decimal as D

import numpy as np
import pytest

from mdbas_b200 import nb, systems
from mdbas_b200.fit_erfc import erfcx_decimal

pytestmark = pytest.mark.gpu

U = 2.0 ** -53
PI = D("3.14159265358979323846264338327950288419716939937510582097494459")
# (alpha, cut-off).  0.5 makes x = 6 exact; the square of 0.2505 is rounded by
# 0.96 u, which e^{-x^2} multiplies by x^2.
RANGE = [(0.34, 12.0), (0.4, 12.0), (0.5, 12.0), (0.2505, 24.0)]


def _pairs(dist, q1=1.0, q2=-1.0):
    """Pairs 64 A apart, the second atom dist along x from the first."""
    m = math.ceil(len(dist) ** (1 / 3) - 1e-9)
    box = 64.0 * m
    site = np.arange(len(dist))
    base = 64.0 * np.stack([site % m, site // m % m, site // (m * m)], 1) + 16.0 - 0.5 * box
    pos = np.repeat(base, 2, axis=0)
    pos[1::2, 0] += dist
    n = len(pos)
    q = np.tile([q1, q2], len(dist))
    return systems.System("pairs", box, *(pos[:, k].copy() for k in range(3)), q, np.zeros(n),
                          np.ones(n), np.ones(n), np.zeros((0, 2), np.int32),
                          np.zeros((0, 3), np.int32))


def _engine(s, alpha, cut_off):
    return nb.Engine(s, precision=0, alpha=alpha, cutOff=cut_off, vdwSwitch=0,
                     exclusions=(np.zeros(s.n + 1, np.int32), np.zeros(0, np.int32)))


def _distances(alpha, cut_off):
    """Multiples of 2^-10 up to x = 6: their squares are exact."""
    last = int(min(cut_off, 6.0 / alpha) * 1024)
    rng = np.random.default_rng(3)
    k = np.concatenate([[2, 3, last - 1, last], 2 ** np.arange(2, 13),
                        np.exp(rng.uniform(np.log(4), np.log(last), 150)).astype(int),
                        rng.integers(1024, last + 1, 250)])
    return k / 1024.0


def _exact(dist, alpha):
    """Per pair: energy and force of unit charges times C."""
    e, f = [], []
    with decimal.localcontext() as ctx:
        ctx.prec = 50
        c, a = D(float(systems.CHARGE_CONST)), D(alpha)
        for r in map(D, dist):
            x = a * r
            g = (-x * x).exp()
            e.append(c * g * erfcx_decimal(x) / r)
            f.append((e[-1] + 2 * c * a / PI.sqrt() * g) / r)
    return e, f


def _off(got, want):
    """Relative errors in u, signed."""
    return np.array([float((D(float(a)) - b) / b) for a, b in zip(got, want)]) / U


@pytest.mark.parametrize("alpha,cut_off", RANGE)
def test_pair_forces(gpu, alpha, cut_off):
    dist = _distances(alpha, cut_off)
    eng = _engine(_pairs(dist), alpha, cut_off)
    eng.build()
    eng.compute()
    fx, fy, fz = eng.forces()
    eng.close()
    assert not fy.any() and not fz.any()
    assert np.array_equal(fx[0::2], -fx[1::2])
    d = _off(fx[0::2], _exact(dist, alpha)[1])
    print(alpha, "force: worst", np.abs(d).max(), "mean", d.mean(), "rms", np.sqrt((d * d).mean()))
    assert np.abs(d).max() <= 23


@pytest.mark.parametrize("alpha,cut_off", RANGE)
def test_pair_adjoint(gpu, alpha, cut_off):
    """dE/dq of an atom without charge is its partner's potential alone."""
    dist = _distances(alpha, cut_off)
    eng = _engine(_pairs(dist, q1=0.0, q2=1.0), alpha, cut_off)
    eng.build()
    got = eng.adjoint()["gq"][0::2]
    eng.close()
    d = _off(got, _exact(dist, alpha)[0])
    print(alpha, "dE/dq: worst", np.abs(d).max(), "mean", d.mean(), "rms",
          np.sqrt((d * d).mean()))
    assert np.abs(d).max() <= 19


@pytest.mark.parametrize("q", [1.0, 2.0 ** -20])
def test_single_pair_energy(gpu, q):
    """The sum over blocks keeps the digits of one weak pair."""
    alpha = 0.5
    dist = np.array([1.0, 4.0, 7.5, 9.0, 10.5, 11.25, 12.0])
    want = [x * D(q) * D(q) for x in _exact(dist, alpha)[0]]
    work = [-x * D(r) * D(q) * D(q) for x, r in zip(_exact(dist, alpha)[1], dist)]
    for r, e, w in zip(dist, want, work):
        eng = _engine(_pairs(np.array([r]), q, q), alpha, 12.0)
        eng.build()
        eng.compute()
        got = eng.energies()
        eng.close()
        assert got["n_pairs"] == 1
        print(q, r, _off([got["elec_direct"]], [e]), _off([got["vir_direct"]], [w]))
        assert abs(_off([got["elec_direct"]], [e])[0]) <= 22
        assert abs(_off([got["vir_direct"]], [w])[0]) <= 23
