"""A halo of negative mass (b0 < 0, accepted by the upload): every sum is linear in b0, so negating the b0 of
every halo negates the deflection, the potential, the convergence and the shear, in every bit (each operation
rounds to nearest)."""
import numpy as np
import pytest

import lenstool_hpc_b200 as lt
from lenstool_hpc_b200 import catalog

pytestmark = pytest.mark.gpu

SMALL, LARGE = catalog.Grid(-90., 95., -80., 85., 61, 43), catalog.Grid(-90., 95., -80., 85., 641, 523)


@pytest.fixture(scope="module")
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    c = lt.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("e", [0.3, 0.97])  # on both sides of the minor axis' change of form, q^2 = 1/16
@pytest.mark.parametrize("ptype", [5, 8, 81])
@pytest.mark.parametrize("grid", [SMALL, LARGE])  # every pair; far halos interpolated
def test_sums_are_odd_in_the_mass(ctx, grid, ptype, e):
    n = 250
    rng = np.random.default_rng(ptype)
    cat = catalog.make_catalog([ptype] * n, rng.uniform(-90., 90., n), rng.uniform(-80., 80., n), rng.uniform(80., 300., n),
                               np.full(n, e), rng.uniform(0., np.pi, n), rng.uniform(0.05, 2., n), rng.uniform(5., 50., n))
    minus = catalog.HaloCatalog(**{f: getattr(cat, f) for f in ("type",) + catalog.FIELDS})
    minus.b0 = -cat.b0
    for precision in ("fp64", "fp64fast"):
        sums = [list(ctx.gradient_grid(c, grid, precision=precision)) + [ctx.potential_grid(c, grid, precision=precision)] +
                list(ctx.hessian_maps(c, grid, ["kappa", "gamma1", "gamma2"], precision=precision).values())
                for c in (cat, minus)]
        for k, (a, b) in enumerate(zip(*sums)):
            assert np.array_equal(a, -b), (precision, k)
