"""Catalogues updated in place and the FP64 sums whose far halos are interpolated: the tiles are chosen by the halos'
spread, which an update from host values refreshes (the planes of a fresh upload bit for bit) and one from device
values cannot (1e-13 of max(|value|, RMS), the bound between any two choices)."""
import numpy as np
import pytest

import lenstool_hpc_b200 as lt
from lenstool_hpc_b200 import bayes as B
from lenstool_hpc_b200 import catalog

from conftest import max_rel_err

pytestmark = pytest.mark.gpu
GRID = catalog.Grid.square(100., 500)


@pytest.fixture(scope="module")
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    c = lt.Context(0)
    yield c
    c.close()


def _planes(ctx, cat):
    return list(ctx.gradient_grid(cat, GRID)) + [ctx.potential_grid(cat, GRID)] + \
        list(ctx.hessian_maps(cat, GRID, ["kappa", "gamma1"], precision="fp64fast").values())


def _placeholder(p):
    q = p.perturbed(np.random.Generator(np.random.PCG64(1)), rel=0.)
    q.position_x[:], q.position_y[:], q.ellipticity[:] = 0., 0., 0.9
    return q


@pytest.mark.parametrize("device", [False, True])
def test_update(ctx, device):
    import torch
    p = catalog.cluster_galaxy_parameters(2, 298, 5)
    fresh, d = ctx.upload(p.catalog()), ctx.upload(_placeholder(p).catalog())
    args = p.update_args()
    d.update(*[torch.tensor(a, device="cuda") for a in args] if device else args)
    for k, (a, b) in enumerate(zip(_planes(ctx, d), _planes(ctx, fresh))):
        assert max_rel_err(a, b) <= 1e-13 if device else np.array_equal(a, b), k


@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("fields", [(B.X, B.Y, B.EMASS, B.THETA), (B.VDISP,)])
def test_bayes_rows(ctx, device, fields):
    import torch
    n = 300
    p = catalog.cluster_galaxy_parameters(2, n - 2, 6)
    model = B.model_from_parameters(p)
    post = ctx.bayes(model, [(f, i) for i in range(0, n, 2) for f in fields])
    rng = np.random.default_rng(2)
    col = {B.X: lambda i: rng.uniform(-30., 30.), B.Y: lambda i: rng.uniform(-30., 30.),
           B.EMASS: lambda i: rng.uniform(0.1, 0.5), B.THETA: lambda i: rng.uniform(0., 180.), B.VDISP: lambda i: 150.}
    rows = np.array([[col[f](i) for i in range(0, n, 2) for f in fields] for _ in range(3)])
    cats = [ctx.upload(_placeholder(p).catalog()) for _ in range(3)]
    post.apply(torch.tensor(rows, device="cuda") if device else rows, cats)
    for r, cat in enumerate(cats):
        q = p.perturbed(np.random.Generator(np.random.PCG64(1)), rel=0.)
        where = {B.X: q.position_x, B.Y: q.position_y, B.EMASS: q.ellipticity, B.THETA: q.ellipticity_angle, B.VDISP: q.vdisp}
        for j, f in enumerate(fields):
            v = rows[r, j::len(fields)]
            where[f][0::2] = v * (np.arccos(-1.) / 180.) if f == B.THETA else v
        fresh = ctx.upload(q.catalog())
        for k, (a, b) in enumerate(zip(_planes(ctx, cat), _planes(ctx, fresh))):
            # the model's step through both ellipticities and the device's cos/sin round apart: 1e-12, as elsewhere
            assert max_rel_err(a, b) <= 1e-12, (r, k)
            if not device and f == B.VDISP:
                assert np.array_equal(a, b), (r, k)
