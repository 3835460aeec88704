"""A cut dPIE whose cut radius is far beyond the field is a PIEMD: its cut term is below rcore/rcut and field/rcut of
the core term.  So the sums of both agree to their rounding (1e-13 of max(|value|, RMS), as the batch's), for cut
radii up to those whose square still is a double; and a core far below the pixels' spacing leaves a singular
ellipse, whose deflection vanishes at its centre."""
import numpy as np
import pytest

import lenstool_hpc_b200 as lt
from lenstool_hpc_b200 import catalog

from conftest import max_rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    c = lt.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("rcut", [1e21, 1e30, 1e36, 1e40, 1e100])
@pytest.mark.parametrize("n, side", [(20, 61), (250, 640)])  # every pair; far halos interpolated
def test_equals_the_uncut_profile(ctx, rcut, n, side):
    rng = np.random.default_rng(n)
    a = (rng.uniform(-90., 90., n), rng.uniform(-90., 90., n), rng.uniform(80., 900., n), rng.uniform(0.01, 0.6, n),
         rng.uniform(0., np.pi, n), rng.uniform(0.05, 9., n))
    cut, uncut = catalog.make_catalog([81] * n, *a, np.full(n, rcut)), catalog.make_catalog([8] * n, *a, np.full(n, 1e3))
    g = catalog.Grid.square(100., side)
    for precision in ("fp64", "fp64fast"):
        sums = [list(ctx.gradient_grid(c, g, precision=precision)) + [ctx.potential_grid(c, g, precision=precision)]
                for c in (cut, uncut)]
        if precision == "fp64fast":
            for s, c in zip(sums, (cut, uncut)):
                s += list(ctx.hessian_maps(c, g, ["kappa", "gamma1", "gamma2"], precision=precision).values())
        for k, (got, want) in enumerate(zip(*sums)):
            assert np.isfinite(got).all() and max_rel_err(got, want) <= 1e-13, (precision, k)


@pytest.mark.parametrize("ptype", [8, 81])
@pytest.mark.parametrize("n, half", [(1, 30), (250, 320)])  # every pair; far halos interpolated
def test_tiny_core(ctx, ptype, n, half):
    rng = np.random.default_rng(n)
    x, y = np.r_[0., rng.uniform(-90., 90., n - 1)], np.r_[0., rng.uniform(-90., 90., n - 1)]
    a = (rng.uniform(80., 900., n), rng.uniform(0.01, 0.6, n), rng.uniform(0., np.pi, n))
    g = catalog.Grid.square(100., 2 * half + 1)
    tiny, small = [np.stack(ctx.gradient_grid(catalog.make_catalog([ptype] * n, x, y, *a, np.full(n, rc),
                                                                   np.full(n, 0.2)), g)) for rc in (1e-40, 1e-30)]
    # 1e-30 is below 1e-16 of the distance to every other pixel
    assert np.isfinite(tiny).all() and max_rel_err(tiny, small) <= 1e-13
    if n == 1:
        assert (tiny[:, half, half] == 0.).all()
