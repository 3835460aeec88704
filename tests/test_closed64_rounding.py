"""Rounding of the FP64 closed forms: the sums of many halos at every pixel, and a cut radius close to the core radius."""
import numpy as np
import pytest

import lenstool_hpc_b200 as lt
from lenstool_hpc_b200 import catalog

from test_closed64 import _reference

pytestmark = pytest.mark.gpu
L = np.longdouble


@pytest.fixture(scope="module")
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    c = lt.Context(0)
    yield c
    c.close()


def _two_norm(got, ref):
    return float(np.sqrt(np.sum((got - ref) ** 2) / np.sum(ref ** 2)))


@pytest.mark.parametrize("n", [700, 2000])
def test_sums_of_every_pair(ctx, n):
    """n like halos on a grid that evaluates every pair: the roundings of chunk sums of 64 and of the total, sqrt(64 / (n / 64)) / 3
    and sqrt(n / 64) / 3 units of 1.1e-16 of the sum (2.1 at n = 2000), and a term's few, 1 / sqrt(n) of them: below
    4e-16.  (One running sum: sqrt(n) / 3, 9.8e-16 at n = 700.)"""
    rng = np.random.default_rng(n)
    cat = catalog.make_catalog([8] * n, rng.uniform(-90., 90., n), rng.uniform(-90., 90., n), np.full(n, 150.),
                               np.full(n, 0.2), rng.uniform(0., np.pi, n), np.full(n, 2.), np.full(n, 100.))
    g = catalog.Grid(-100., 100., -100., 100., 47, 45)
    px, py = g.coords()
    ref = L(0)
    for i in range(n):
        ref = ref + _reference(8, cat.ellipticity_potential[i], cat.b0[i], cat.rcore[i], cat.rcut[i], cat.ellipticity_angle[i],
                               px - L(cat.position_x[i]), py - L(cat.position_y[i]))[3]
    kappa = ctx.hessian_maps(cat, g, ["kappa"], precision="fp64fast")["kappa"].ravel()
    assert _two_norm(kappa, ref) <= 4e-16


@pytest.mark.parametrize("precision", ["fp64", "fp64fast"])
@pytest.mark.parametrize("ratio", [1e-9, 1e-5, 0.3, 0.99, 1.01])
def test_cut_radius_close_to_the_core(ctx, precision, ratio):
    """rcut = rcore (1 + ratio): the core minus the cut term, taken without cancellation (in extended precision from the
    same radii), to the 7e-14 of a lone halo (test_closed64.py)."""
    e, b0, rc, theta = 0.2, 2., 0.7, 0.4
    rcut = rc * (1. + ratio)
    n = np.ones(1)
    cat = catalog.HaloCatalog(type=np.array([81], np.int32), position_x=0 * n, position_y=0 * n, b0=b0 * n,
                              ellipticity_angle=theta * n, anglecos=np.cos(theta) * n, anglesin=np.sin(theta) * n,
                              ellipticity_potential=e * n, rcore=rc * n, rcut=rcut * n, dlsds=n)
    g = catalog.Grid(-5., 5., -5., 4.5, 46, 31)
    px, py = g.coords()
    c, s = L(np.cos(theta)), L(np.sin(theta))
    u, v = px * c + py * s, py * c - px * s
    E, R, T = L(e), L(rc), L(rcut)
    q, k = (1 - E) / (1 + E), 2 * np.sqrt(E) / (1 + E)
    A, S, C, d = L(b0) * (1 - E) * T / (T - R), (1 + E) * R, (1 + E) * T, (1 + E) * (R - T)
    pc, pt = np.sqrt(q * q * (S * S + u * u) + v * v), np.sqrt(q * q * (C * C + u * u) + v * v)
    dp = q * q * d * (S + C) / (pc + pt)
    au = A / k * np.arctan(-k * u * (dp + d) / ((pc + S) * (pt + C) + k * k * u * u))
    av = A / k * np.arctanh(-k * v * (dp + q * q * d) / ((pc + q * q * S) * (pt + q * q * C) - k * k * v * v))
    rx, ry = au * c - av * s, au * s + av * c
    amp = np.hypot(rx, ry)
    ax, ay = ctx.gradient_grid(cat, g, precision=precision)
    assert np.max(np.abs(ax.ravel() - rx) / amp) <= 7e-14 and np.max(np.abs(ay.ravel() - ry) / amp) <= 7e-14
