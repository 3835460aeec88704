"""Every two-pixel shape of the LT_FP32C kernels (one record and two at a time, packed and scalar, each stage size) and
the shapes that the default context picks on small and large grids, against the one-pixel shape, which takes the
scalar form record by record.  All round every operation alike, so the planes are equal bit for bit wherever no FP64
disc is near (the halos lie outside the field)."""
import numpy as np
import pytest

import lenstool_hpc_b200 as lt
from lenstool_hpc_b200 import catalog

pytestmark = pytest.mark.gpu

SHAPES = [None, (2, 2, 256, 128), (2, 1, 256, 32), (2, 2, 128, 64), (2, 3, 128, 32), (2, 4, 128, 64), (2, 4, 128, 128)]


def _maps(cat, g, config):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    with lt.Context(0) as ctx:
        for sums in ("deflection", "hessian", "potential", "lens") if config else ():
            ctx.set_kernel_config("fp32c", sums, *config)
        h = ctx.upload(cat)
        ax, ay = ctx.gradient_grid(h, g, precision="fp32c")
        out = {"ax": ax, "ay": ay, "psi": ctx.potential_grid(h, g, precision="fp32c")}
        out.update(ctx.hessian_maps(h, g, ["kappa", "gamma1", "gamma2"], precision="fp32c", kmap=True))
        for k, v in ctx.lens_maps(h, g, precision="fp32c", dlsds=1., which=("gamma1", "gamma2", "psi")).items():
            out["lens " + k] = v
        return out


# grids of under a warp a scheduler; above the small grids' limits (4 warps, lens maps 1.6) with ragged edges; of
# more than a wave of tiles
@pytest.mark.parametrize("grid", [(65, 41), (331, 203), (641, 403)])
@pytest.mark.parametrize("types, n", [([81], 65), ([8], 33), ([5], 130), ([5, 8, 81], 257)])
def test_shapes_are_equal(grid, types, n):
    rng = np.random.default_rng(n)
    cat = catalog.make_catalog(sorted((types * n)[:n]), rng.uniform(-200., -120., n), rng.uniform(-90., 90., n),
                               rng.uniform(80., 200., n), rng.uniform(0.05, 0.5, n), rng.uniform(0., np.pi, n),
                               rng.uniform(0.05, 0.2, n), rng.uniform(1., 300., n), dlsds=rng.choice([0.5, 0.8], n))
    nx, ny = grid
    g = catalog.Grid(-100., 100., -80., 90., nx, ny)
    want = _maps(cat, g, (1, 2, 256, 64))
    assert np.array_equal(want["lens psi"], want["psi"])
    for config in SHAPES:
        got = _maps(cat, g, config)
        for k in want:
            assert np.array_equal(got[k], want[k]), (config, k)
