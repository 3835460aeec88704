"""Batches (lenstool-hpc_b200/csrc/lt_queue.cu): tiles claimed by addition, flagged pixels gathered over
the tiles of a request.  The maps are those of the single calls bit for bit and every flagged pixel is
recomputed once, whatever remains on a CTA's list when its request ends."""
import numpy as np
import pytest

import lenstool_hpc_b200 as lt
from lenstool_hpc_b200 import catalog

pytestmark = pytest.mark.gpu

# one tile, ragged tiles, fewer tiles than CTAs, several tiles a CTA (its list passes 512 pixels)
SIDES = [(33, 7), (64, 8), (129, 65), (257, 300), (700, 650), (1024, 1024)]


@pytest.fixture(scope="module")
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    c = lt.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("halos", [3, 200])
@pytest.mark.parametrize("order", ["large first", "repeated"])
def test_batch_equals_single_calls(ctx, halos, order):
    import torch
    cat = catalog.cluster_galaxy_catalog(2, halos - 2, 5)
    cat.type = np.sort(np.random.default_rng(halos).choice(np.array([5, 8, 81, 81], np.int32), halos))
    cat = ctx.upload(cat)
    sides = SIDES if order == "large first" else [SIDES[3]] * 9 + [SIDES[0]] * 40
    grids = [catalog.Grid(-60., 60., -60. * ny / nx, 60. * ny / nx, nx, ny) for nx, ny in sides]
    new = lambda g: {k: torch.full((g.ny, g.nx), np.nan, dtype=torch.float64, device="cuda") for k in ("kappa", "mu")}
    want, got = [new(g) for g in grids], [new(g) for g in grids]
    ctx.recompute_count()
    for g, o in zip(grids, want):
        ctx.hessian_maps(cat, g, ["kappa", "mu"], precision="fp32c", dlsds=0.7, out=[o["kappa"], o["mu"]])
    ctx.synchronize()
    flagged = ctx.recompute_count()
    b = ctx.batch([lt.Request(cat, g, o, dlsds=0.7) for g, o in zip(grids, got)], precision="fp32c")
    for _ in range(2):
        b.launch()
        ctx.synchronize()
        assert ctx.recompute_count() == flagged
    b.destroy()
    assert halos < 200 or flagged > 0
    for g, w, o in zip(grids, want, got):
        for k in w:
            assert torch.equal(w[k], o[k]), (g.nx, g.ny, k)
