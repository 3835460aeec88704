"""The correctly rounded quotients and square roots of the reference-order Hessian
(lenstool-hpc_b200/csrc/lt_profiles64.cuh: quot, rcp_rn, sqrt_rn): the same steps on every
operand of small precisions (CPU), and the kernel on operands they do not cover (GPU)."""
from fractions import Fraction as F
from math import isqrt

import numpy as np
import pytest

import lenstool_hpc_b200 as lt
from lenstool_hpc_b200 import catalog


def _rn(x, p):
    """x (a Fraction) rounded to p bits, ties to even."""
    if x == 0:
        return F(0)
    n, d = abs(x.numerator), x.denominator
    k = p - 1 - (n.bit_length() - d.bit_length())
    scale = lambda k: (n << k, d) if k >= 0 else (n, d << -k)  # noqa: E731
    a, b = scale(k)
    if a < b << (p - 1):
        k += 1
    a, b = scale(k)
    q, r = divmod(a, b)
    q += 2 * r > b or (2 * r == b and q & 1)
    return (-1 if x < 0 else 1) * F(q) * (F(1, 1 << k) if k >= 0 else F(1 << -k))


def _fma(a, b, c, p):
    return _rn(a * b + c, p)


def _root(x, p):
    """sqrt(x) with a sticky bit beyond p."""
    s = 4 * p + 40
    v = isqrt((x.numerator << (2 * s)) // x.denominator)
    f = F(v, 1 << s)
    return f if f * f == x else f + F(1, 1 << (s + 3))


def _ulp(y, p):
    e = 0
    while y >= 2:
        y, e = y / 2, e + 1
    while y < 1:
        y, e = y * 2, e - 1
    return F(2) ** (e - p + 1)


@pytest.mark.parametrize("p", [6, 7])
def test_quotients_of_every_operand(p):
    one = 1 << (p - 1)
    for m in range(one, 2 * one):
        b = F(m, one)
        y = _rn(1 / b, p)
        for n in range(one, 2 * one):
            a = F(n, one)
            q = _rn(a * y, p)
            assert _fma(_fma(-q, b, a, p), y, q, p) == _rn(a / b, p), (m, n)


@pytest.mark.parametrize("p", [8, 10])
def test_reciprocals_of_every_operand(p):
    one = 1 << (p - 1)
    for m in range(one, 2 * one - 1):  # 2 one - 1: all ones, not covered
        b = F(m, one)
        r = _rn(1 / b, p)
        u = _ulp(r, p)
        for y in (r - u, r, r + u):
            if abs(y - 1 / b) <= u * F(65, 128):
                assert _fma(_fma(-b, y, F(1), p), y, y, p) == r, m


@pytest.mark.parametrize("p", [7, 8, 9])
def test_square_roots_of_every_operand(p):
    one = 1 << (p - 1)
    for m in range(one, 2 * one):
        for x in (F(m, one), 2 * F(m, one)):
            s = _rn(_root(x, p), p)
            if s == _rn(s, p) and (s / _ulp(s, p)) == 2 * one - 1 or m >= 2 * one - 2:
                continue  # a root of all ones, or x ending in 11..10, 11..11: not covered
            y0 = _rn(1 / _root(x, p), p)
            u = _ulp(y0, p)
            for y in (y0 - u, y0, y0 + u):
                if not (max(y - u, 0) ** 2 * x <= 1 <= (y + u) ** 2 * x):
                    continue  # further than an ulp from 1/sqrt(x)
                g = _rn(x * y, p)
                g1 = _fma(_fma(-g, g, x, p), y / 2, g, p)
                y1 = _fma(_fma(-g1, y, F(1), p), y, y, p)
                w = _fma(_fma(-g1, g1, x, p), y1 / 2, g1, p)
                assert w == s, (m, x)
                assert _fma(_fma(-w, y1, F(1), p), y1, y1, p) == _rn(1 / s, p), (m, x)


@pytest.mark.gpu
@pytest.mark.parametrize("ptype", [81, 8])
def test_uncovered_operands_take_the_ieee_steps(oracle_lib, ptype):
    """Divisors whose significand ends in 32 ones, zero, tiny and huge offsets: bit for bit the
    oracle's Hessian.  At u = x, v = 2 r sqrt(e) the second divisor is x^2 rounded."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    ctx = lt.default_context()
    e, rc, rcut = 0.25, 0.5, 20.
    one = np.ones(1)
    cat = catalog.HaloCatalog(type=np.array([ptype], np.int32), position_x=0 * one, position_y=0 * one, b0=2. * one,
                              ellipticity_angle=0 * one, anglecos=one, anglesin=0 * one,
                              ellipticity_potential=e * one, rcore=rc * one, rcut=rcut * one, dlsds=one)
    pts = []
    for top in range(400):
        want = np.array([(0x40100000 + 977 * top) << 32 | 0xffffffff], np.uint64).view(np.float64)[0]
        x = np.sqrt(want)
        for c in (x, np.nextafter(x, 0.), np.nextafter(x, 9.)):
            if (np.float64(c * c).view(np.uint64) & np.uint64(0xffffffff)) == 0xffffffff:
                pts.append((float(c), 2 * rc * np.sqrt(e)))
    assert len(pts) >= 50
    pts += [(0., 3.), (1e-300, 2.), (-1e-160, 1.), (0., 0.), (2., 0.), (3., -1e-200), (1e150, 2.), (2., 1e180), (0., 1.)]
    px, py = (np.array([p[i] for p in pts]) for i in (0, 1))
    want = oracle_lib.hess_points(cat, px, py)
    kinds = ["hess_a", "hess_b", "hess_c", "hess_d"]
    for i, (x, y) in enumerate(pts):
        # two pixels a thread: the second one is an ordinary pixel
        m = ctx.hessian_maps(cat, catalog.Grid(x, x + 1., y, y + 1., 2, 1, dx=max(1., abs(x)), dy=1.), kinds)
        for k, name in enumerate(kinds):
            assert np.array_equal(m[name][0, 0], want[k][i], equal_nan=True), (x, y, name)
