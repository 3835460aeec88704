"""The FP32C pair loop of two pixels a thread evaluates a cut dPIE in packed form, and in small CTAs two
records of any type at a time; with one pixel a thread it takes the scalar form, record by record.  All
round every operation alike, so the planes of the shapes are equal wherever no FP64 disc is near (a warp
of each shape covers another box, and a disc sends the whole box to FP64)."""
import numpy as np
import pytest

import lenstool_hpc_b200 as lt
from lenstool_hpc_b200 import catalog

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    c = lt.Context(0)
    yield c
    c.close()


def _maps(ctx, cat, g, config):
    for sums in ("deflection", "hessian", "potential", "lens"):
        ctx.set_kernel_config("fp32c", sums, *config)
    h = ctx.upload(cat)
    ax, ay = ctx.gradient_grid(h, g, precision="fp32c")
    out = {"ax": ax, "ay": ay, "psi": ctx.potential_grid(h, g, precision="fp32c")}
    out.update(ctx.hessian_maps(h, g, ["kappa", "gamma1", "gamma2"], precision="fp32c"))
    for k, v in ctx.lens_maps(h, g, precision="fp32c", dlsds=1., which=("kappa", "gamma1", "psi")).items():
        out["lens " + k] = v
    return out


@pytest.mark.parametrize("n", [1, 7, 8, 9, 63, 65, 130, 257])
@pytest.mark.parametrize("grid", [(96, 64), (65, 41), (1, 7), (130, 1)])
@pytest.mark.parametrize("types", [[81], [8], [5], [5, 8, 81]])
def test_packed_equals_scalar(ctx, n, grid, types):
    rng = np.random.default_rng(n)
    # every halo and its disc left of the field
    cat = catalog.make_catalog(sorted((types * n)[:n]), rng.uniform(-200., -120., n), rng.uniform(-90., 90., n),
                               rng.uniform(80., 200., n), rng.uniform(0.05, 0.5, n), rng.uniform(0., np.pi, n),
                               rng.uniform(0.05, 0.2, n), rng.uniform(1., 300., n))
    nx, ny = grid
    g = catalog.Grid(-100., 100., -80., 90., nx, ny, dx=200. / 96, dy=170. / 64)
    a, b = _maps(ctx, cat, g, (1, 2, 256, 64)), _maps(ctx, cat, g, (2, 2, 256, 64))
    for k in a:
        assert np.array_equal(a[k], b[k]), k
    # the fused maps, and other stage sizes (chunks of 8 halos' blocks in the same order)
    assert np.array_equal(b["lens kappa"], b["kappa"]) and np.array_equal(b["lens psi"], b["psi"])
