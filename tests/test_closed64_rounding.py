"""Rounding of the FP64 closed forms: the sums of many halos at every pixel."""
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
