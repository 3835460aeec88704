"""The interpolated deflection of both FP64 precisions where a comparison of the two with one another says nothing (they
take the same kernel): the 1000-halo workload field against extended precision, the chi2 against the oracle."""
import numpy as np
import pytest

import lenstool_hpc_b200 as lt
from lenstool_hpc_b200 import catalog
from lenstool_hpc_b200.images import generate_systems

from conftest import max_rel_err
from test_closed64 import _reference

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    c = lt.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("precision", ["fp64", "fp64fast"])
def test_deflection_of_the_workload(ctx, precision):
    """1e-13 of max(|value|, RMS): the terms' own 7e-14 at most (test_closed64.py), truncation below 3e-14 of a term at
    the far limit only, and the sums' rounding, taken over at most 128 terms at once."""
    cat, g0 = catalog.workload("maps_1000h_4096")
    g = catalog.Grid(g0.xmin, g0.xmax, g0.ymin, g0.ymax, 768, 768)
    idx = np.random.default_rng(2).choice(g.npix, 1500, replace=False)
    px, py = g.coords(idx)
    want = [np.zeros(idx.size, np.longdouble) for _ in range(2)]
    for i in range(cat.n):
        t = _reference(int(cat.type[i]), cat.ellipticity_potential[i], cat.b0[i], cat.rcore[i], cat.rcut[i],
                       cat.ellipticity_angle[i], px - np.longdouble(cat.position_x[i]), py - np.longdouble(cat.position_y[i]))
        want = [want[0] + t[0], want[1] + t[1]]
    for got, ref in zip(ctx.gradient_grid(cat, g, precision=precision), want):
        assert max_rel_err(got.ravel()[idx], ref) <= 1e-13


@pytest.mark.parametrize("precision", ["fp64", "fp64fast"])
@pytest.mark.parametrize("n", [512, 900])
def test_chi2_matches_oracle(ctx, oracle_lib, precision, n):
    """The same images found and chi2 to 1e-12, as deflections 1e-12 apart give it away from the triangles' edges."""
    frame = (-100., 100., -100., 100.)
    cat = catalog.cluster_galaxy_catalog(2, 198, 20261203)
    ic = int(np.argmax(cat.b0))
    s = generate_systems(lambda bx, by, dr: ctx.delense(cat, frame, 1024, bx, by, dr), 10, 21, dr=0.6,
                         centre=(cat.position_x[ic], cat.position_y[ic]), source_radius=8.)
    model = catalog.perturb_catalog(cat, np.random.Generator(np.random.PCG64(4)))
    chi, found = ctx.chi2(model, frame, n, s, precision=precision)
    ref = oracle_lib.chi2(model, frame, n, s.nimg, s.x, s.y, s.dr)
    assert found == ref["images_found"]
    assert abs(chi - ref["chi2"]) <= 1e-12 * max(1., abs(ref["chi2"]))
