"""The FP64 fits of the damped Coulomb terms (terms.cuh, dsf_terms) against
40-digit arithmetic: the coefficients as the source has them, so that a digit
lost or swapped shows, and the whole evaluation with every operation rounded
as the kernel rounds it.

The interpolants' own errors are 1.6e-17 (exp) and 3.7e-17 (R); the bounds
below add the coefficients' rounding.  Rounded throughout, the Gaussian has one
addition at the end (half an ulp, 1.11e-16, at most 0.7e-16 rms) after terms a third
as large, and erfc the product of two such values with u's rounding, which R
changes by up to twice: 3 x 0.6e-16 rms at most.
"""
import decimal
import os
import re
from fractions import Fraction

import numpy as np
import pytest

from conftest import ROOT

D = decimal.Decimal
SRC = open(os.path.join(ROOT, "capacmd_b200", "csrc", "terms.cuh")).read()
BODY = SRC[SRC.index("dsf_terms(const double (&alpha)[W]"):]
BODY = BODY[:BODY.index("__device__ __forceinline__ Dsf dsf_terms(double alpha, double r2)")]


@pytest.fixture(autouse=True)
def _digits():
    with decimal.localcontext() as ctx:
        ctx.prec = 40
        yield


def _chains():
    """The Horner chains, highest degree first: exp's odd and even, R's odd and even."""
    out = []
    for text, var in zip(BODY.split("// R(x)"), ("f2", "u2")):
        for name in "ab":
            head = re.search(r"%s\[w\] = fma\((\S+), %s\[w\], (\S+)\);" % (name, var), text)
            tail = re.findall(r"chain\(%s, %s, (\S+)\);" % (name, var), text)
            out.append([float(c) for c in head.groups()] + [float(c) for c in tail])
    assert [len(c) for c in out] == [5, 5, 9, 10]
    return out


def _erfc(x):
    """erfc of a Decimal in [0, 27]."""
    isp = D("0.56418958354775628694807945156077258584405")
    if x < 3:
        t = s = x
        k = 0
        while abs(t) > D("1e-38"):
            k += 1
            t *= -x * x / k
            s += t / (2 * k + 1)
        return 1 - 2 * isp * s
    f = D(0)
    for k in range(300, 0, -1):
        f = D(k) / 2 / (x + f)
    return (-x * x).exp() * isp / (x + f)


def _horner(c, t):
    s = D(0)
    for k in c:
        s = s * t + D(k)
    return s


def test_exp_interpolant():
    odd, even = _chains()[:2]
    for f in np.linspace(-0.34657, 0.34657, 201):
        f = D(float(f))
        g = 1 + f + f * f * (_horner(odd, f * f) * f + _horner(even, f * f))
        assert abs(g / f.exp() - 1) < D("3e-17")


def test_scaled_erfc_interpolant():
    odd, even = _chains()[2:]
    for x in np.linspace(0.0, 5.0, 251):
        x = D(float(x))
        u = (x - D("3.5")) / (x + D("3.5"))
        R = _horner(odd, u * u) * u + _horner(even, u * u)
        assert abs(R / (_erfc(x) * (x * x).exp()) - 1) < D("6e-17")


def test_beyond_the_fitted_range():
    """The metal pairs' x is held below 26: erf = 1 - erfc there is right to far
    below a rounding."""
    odd, even = _chains()[2:]
    for x in np.linspace(5.0, 26.0, 211):
        x = D(float(x))
        u = (x - D("3.5")) / (x + D("3.5"))
        ec = (-x * x).exp() * (_horner(odd, u * u) * u + _horner(even, u * u))
        assert abs(ec - _erfc(x)) < D("1e-24")


def fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def _approx(v):
    """A value with 20 bits after the leading one, as the hardware's approximations have at least."""
    return float((np.array([v]).view(np.int64) & np.int64(-1 << 32)).view(np.float64)[0])


def _dsf(alpha, r2, chains, close=True):
    odd_e, even_e, odd, even = chains
    hi, lo = (float.fromhex(v) for v in ("0x1.62e42fef00000p-1", "0x1.473de6af278edp-34"))
    assert "0x1.62e42fef00000p-1" in BODY and "0x1.473de6af278edp-34" in BODY

    def horner(c, t):
        s = c[0]
        for k in c[1:]:
            s = fma(s, t, k)
        return s

    y = _approx(r2 ** -0.5)
    e = fma(-(r2 * y), y, 1.0)
    r = r2 * fma(y * e, fma(0.375, e, 0.5), y)
    al2 = alpha * alpha
    x2 = al2 * r2
    n = fma(x2, -1.4426950408889634, 6755399441055744.0) - 6755399441055744.0
    f = fma(n, -lo, fma(n, -hi, -x2)) - fma(al2, r2, -x2)
    f2 = f * f
    eg = (1.0 + fma(f2, fma(horner(odd_e, f2), f, horner(even_e, f2)), f)) * 2.0 ** n
    z = fma(alpha, r, 3.5)
    dz = fma(alpha, r, 3.5 - z)
    y = _approx(1.0 / z)
    e = fma(-z, y, 1.0)
    if close:
        y = fma(y, e, y)
        q = 7.0 * y
        u = fma(-y, fma(-dz, q, fma(-z, q, 7.0)), 1.0 - q)
    else:
        u = fma(-7.0, fma(y, fma(e, e, e), y), 1.0)
    u2 = u * u
    a, b = horner(odd, u2), horner(even, u2)
    R = fma(a, u, b)
    return eg, fma(eg, R, eg * fma(a, u, b - R)) if close else eg * R


@pytest.mark.parametrize("alpha,r_max", [(2.0, 1.2), (4.0, 1.2), (0.75, 6.6)])
def test_rounded_evaluation(alpha, r_max):
    # powers of two and 3/4: alpha^2 is exact, and what is left is the evaluation
    rng = np.random.default_rng(8)
    chains = _chains()
    err = []
    for r2 in rng.uniform(0.1, r_max, 300) ** 2:
        eg, ec = _dsf(alpha, float(r2), chains)
        x2 = D(alpha) * D(alpha) * D(float(r2))
        err.append((float(D(eg) / (-x2).exp() - 1), float(D(ec) / _erfc(x2.sqrt()) - 1)))
    rms, most = np.sqrt((np.array(err) ** 2).mean(0)), np.abs(err).max(0)
    assert rms[0] < 0.8e-16 and most[0] < 2.0e-16, (rms, most)
    assert rms[1] < 1.8e-16 and most[1] < 6.0e-16, (rms, most)


def test_rounded_erf_of_the_metal_blocks():
    """1 - erfc beyond x = 1.5, in the form without the remainders: half an ulp of
    the subtraction (5.6e-17) and erfc's error, at most 0.034 x 8e-16."""
    rng = np.random.default_rng(9)
    chains = _chains()
    err = []
    for x in rng.uniform(1.5, 6.0, 300):
        alpha = 0.5
        r2 = float((x / alpha) ** 2)
        ec = _dsf(alpha, r2, chains, close=False)[1]
        err.append(float(D(1.0 - ec) - (1 - _erfc((D(alpha) * D(alpha) * D(r2)).sqrt()))))
    assert np.abs(err).max() < 8.4e-17, np.abs(err).max()
