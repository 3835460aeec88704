"""The FP64 closed forms (lenstool-hpc_b200/csrc/lt_closed64.cuh): the tables against decimal
arithmetic (CPU), the kernels against the same forms in extended precision (GPU)."""
import pathlib
import re
from decimal import Decimal, getcontext

import numpy as np
import pytest

import lenstool_hpc_b200 as lt
from lenstool_hpc_b200 import catalog

HEADER = pathlib.Path(__file__).resolve().parent.parent / "lenstool-hpc_b200" / "csrc" / "lt_closed64.cuh"


def _table(name):
    text = HEADER.read_text()
    body = text[text.index(f"{name}["):]
    body = body[body.index("{") + 1:body.index("}")]
    return [float.fromhex(x) for x in re.findall(r"-?0x[0-9a-f.]+p[-+]\d+", body)]


def _atan(x):
    n = 0
    while x > Decimal("0.1"):
        x, n = x / (1 + (1 + x * x).sqrt()), n + 1
    s, t, k = Decimal(0), x, 1
    while abs(t) > Decimal(10) ** -45:
        s, t, k = s + t / k, -t * x * x, k + 2
    return s * 2 ** n


def test_tables_are_correctly_rounded():
    getcontext().prec = 50
    pi = 4 * _atan(Decimal(1))
    a = [_atan(Decimal(j) / 64) for j in range(65)]
    assert _table("kAtanTab") == [float(x) for x in a] + [float(pi / 2 - x) for x in a]
    assert _table("kLogTab") == [float((1 + Decimal(j) / 64).ln()) for j in range(64)]


def _reference(ptype, e, b0, rc, rcut, theta, x, y):
    """Deflection, potential, convergence and shear of one halo at the origin, extended precision."""
    L = np.longdouble
    e, b0, rc, rcut = L(e), L(b0), L(rc), L(rcut)
    c, s = L(np.cos(theta)), L(np.sin(theta))
    x, y = x.astype(L), y.astype(L)
    u, v = x * c + y * s, y * c - x * s
    q, k = (1 - e) / (1 + e), 2 * np.sqrt(e) / (1 + e)
    A = b0 * (1 - e) * (rcut / (rcut - rc) if ptype == 81 else 1)
    au = av = p = kap = a = b = L(0)
    for r, sg in ((rc, 1), (rcut, -1))[:2 if ptype == 81 else 1]:
        S = (1 + e) * r
        psi = np.sqrt(q * q * (S * S + u * u) + v * v)
        E = A / 2 / psi / ((1 + q * q) * S * S + 2 * S * psi + u * u + v * v)
        kap, a, b = kap + sg * A / 2 / psi, a + sg * E * ((q * q - 1) * S * S + v * v - u * u), b - sg * 2 * E * u * v
        du, dv = A / k * np.arctan(k * u / (psi + S)), A / k * np.arctanh(k * v / (psi + q * q * S))
        t = (u * u + v * v + 2 * S * (q * q * u * u + v * v) / (psi + q * S)) / (4 * r * r)
        au, av, p = au + sg * du, av + sg * dv, p + sg * (u * du + v * dv - A * S / 2 * np.log1p(t))
    c2, s2 = c * c - s * s, 2 * s * c
    return au * c - av * s, au * s + av * c, p, kap, a * c2 - b * s2, a * s2 + b * c2


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp64fast"])
@pytest.mark.parametrize("ptype", [81, 8])
@pytest.mark.parametrize("e", [1e-5, 1e-3, 0.2, 0.55, 0.599, 0.601, 0.8])
def test_lone_halo_against_extended_precision(ptype, e, precision):
    """One halo, from a tenth of its core to a hundred cut radii, each value relative to its
    own size (the shear to kappa + |shear|).  About 40 roundings of 1.1e-16, those of the
    arc tangent's and the logarithm's denominators amplified up to 1/q^2 = 16 at the switch
    of forms (e = 0.6): 7e-14; above it q itself, 1 - e rounded, costs 1/(1 - e) more."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    ctx = lt.default_context()
    tol = 7e-14
    for rc, rcut, theta in ((0.1, 0.5, 0.3), (0.1, 30., 2.), (5., 5.5, 1.1)):
        n = np.ones(1)
        cat = catalog.HaloCatalog(type=np.array([ptype], np.int32), position_x=0 * n, position_y=0 * n, b0=2. * n,
                                  ellipticity_angle=theta * n, anglecos=np.cos(theta) * n, anglesin=np.sin(theta) * n,
                                  ellipticity_potential=e * n, rcore=rc * n, rcut=rcut * n, dlsds=n)
        for half in (0.1 * rc, rc, 3 * rcut, 100 * rcut):
            g = catalog.Grid(-half, half, -half, 0.9 * half, 46, 31)
            px, py = g.coords()
            rx, ry, rp, rk, r1, r2 = _reference(ptype, e, 2., rc, rcut, theta, px, py)
            ax, ay = ctx.gradient_grid(cat, g, precision=precision)
            psi = ctx.potential_grid(cat, g, precision=precision)
            amp = np.hypot(rx, ry)
            assert np.max(np.abs(ax.ravel() - rx) / amp) <= tol and np.max(np.abs(ay.ravel() - ry) / amp) <= tol
            assert np.max(np.abs(psi.ravel() - rp) / np.abs(rp)) <= tol
            if precision == "fp64fast" and half <= 3 * rcut:
                # the core - cut differences are taken directly: relative to the core term,
                # (r/rcut)^2/2 above the difference at most (5 at 3 rcut)
                m = ctx.hessian_maps(cat, g, ["kappa", "gamma1", "gamma2"], precision=precision)
                size = np.abs(rk) + np.hypot(r1, r2)
                for got, ref in zip(m.values(), (rk, r1, r2)):
                    assert np.max(np.abs(got.ravel() - ref) / size) <= tol


@pytest.mark.gpu
def test_potential_at_a_centre():
    """pi05 is 0/0 at a halo's centre: NaN there, as in the reference; the deflection vanishes."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    cat = catalog.make_catalog([81], [1.], [2.], [200.], [0.3], [0.4], [0.1], [10.])
    g = catalog.Grid(0., 2., 1., 3., 3, 3)
    ctx = lt.default_context()
    psi = ctx.potential_grid(cat, g)
    assert np.isnan(psi[1, 1]) and np.isfinite(np.delete(psi.ravel(), 4)).all()
    ax, ay = ctx.gradient_grid(cat, g)
    assert ax[1, 1] == 0. and ay[1, 1] == 0.
