"""Derivation of the FP32 erfc used by the mixed-precision pair kernel.

Form (Abramowitz & Stegun 7.1.26, refitted here):

    erfc(x) ~= t * P(t) * exp(-x^2),   t = 1 / (1 + p x),   x in [0, 6],

with P of degree 7.  p and the coefficients minimise the maximum RELATIVE
error of t*P(t) against the scaled complementary error function
erfcx(x) = erfc(x) exp(x^2) (scipy.special.erfcx, FP64) on 20,001 points:
p by a bounded scalar search, the coefficients by Lawson's iteratively
reweighted least squares toward the minimax solution.  Running this script
prints the constants compiled into csrc/pair_fp32.cu and the fit's maximum
relative error (2.4e-8).

fit64 derives the FP64 form of csrc/real64.cuh: (x + 3) erfcx(x) as a
polynomial of degree 18 in t = (x - 3) / (x + 3), x in [0, 6], by Chebyshev
interpolation; the map is that of Shepherd and Laframboise (Math. Comp. 36
(1981) 249), who take (1 + 2 x) erfcx(x) over [0, inf).  erfcx comes from the power series of erf (x < 5) or the
continued fraction of erfc, in 70-digit decimal arithmetic; the interpolation
error is 1.9e-17 relative.
"""
import math
from decimal import Decimal as D
from decimal import localcontext

import numpy as np
from scipy.optimize import minimize_scalar
from scipy.special import erfcx

X0, X1, DEG = 0.0, 6.0, 7


def fit(p, deg=DEG, iters=60):
    x = np.linspace(X0, X1, 20001)
    t = 1.0 / (1.0 + p * x)
    y = erfcx(x)
    a = np.stack([t ** (k + 1) for k in range(deg + 1)], 1)
    w = 1.0 / y
    for _ in range(iters):
        c, *_ = np.linalg.lstsq(a * w[:, None], y * w, rcond=None)
        err = (a @ c - y) / y
        w = w * (np.abs(err) + 1e-3 * np.abs(err).max()) ** 0.5
        w /= w.max() / (1.0 / y).max()
    err = (a @ c - y) / y
    return float(np.abs(err).max()), c


def erfcx_decimal(x: D) -> D:
    root_pi = D("3.14159265358979323846264338327950288419716939937510582097494459230781640628620900").sqrt()
    if x < 5:
        # erf(x) = 2/sqrt(pi) exp(-x^2) sum 2^n x^(2n+1) / (2n+1)!!
        s, t, n = D(0), x, 0
        while abs(t) > D(10) ** -68:
            s += t
            n += 1
            t = t * 2 * x * x / (2 * n + 1)
        return (x * x).exp() - 2 / root_pi * s
    f = x
    for k in range(1200, 0, -1):
        f = x + (D(k) / 2) / f
    return 1 / root_pi / f


def fit64(k=D(3), x1=D(6), deg=18):
    """(coefficients, maximum relative error) of (x + k) erfcx(x) in t."""
    with localcontext() as ctx:
        ctx.prec = 70
        lo, hi, n = D(-1), (x1 - k) / (x1 + k), deg + 1
        ts = [(lo + hi) / 2 + (hi - lo) / 2 * D(math.cos(math.pi * (i + 0.5) / n))
              for i in range(n)]
        c = []
        for t in ts:
            x = k * (1 + t) / (1 - t)
            c.append(erfcx_decimal(x) * (x + k))
        for j in range(1, n):  # divided differences, then monomials
            for i in range(n - 1, j - 1, -1):
                c[i] = (c[i] - c[i - 1]) / (ts[i] - ts[i - j])
        p = [D(0)]
        for i in range(n - 1, -1, -1):
            q = [D(0)] * (len(p) + 1)
            for m, v in enumerate(p):
                q[m + 1] += v
                q[m] -= v * ts[i]
            q[0] += c[i]
            p = q
        p = p[:n]
        worst = 0.0
        for i in range(1, 240):
            x = x1 * D(i) / 240
            t, s = (x - k) / (x + k), D(0)
            for v in reversed(p):
                s = s * t + v
            worst = max(worst, abs(float(s / (x + k) / erfcx_decimal(x) - 1)))
        return [float(v) for v in p], worst


def main():
    res = minimize_scalar(lambda p: fit(p, DEG, 20)[0], bounds=(0.2, 1.5), method="bounded",
                          options={"xatol": 1e-5})
    e, c = fit(res.x, DEG, 120)
    print(f"p = {res.x:.9e}f")
    for k, v in enumerate(c):
        print(f"c{k} = {v:.9e}f")
    print(f"max relative error on [{X0}, {X1}]: {e:.3e}")
    c64, e64 = fit64()
    for k, v in enumerate(c64):
        print(f"d{k} = {v!r}")
    print(f"max relative error of the FP64 form on [0, 6]: {e64:.3e}")


if __name__ == "__main__":
    main()
