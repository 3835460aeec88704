"""FP64 sums with the far halos interpolated over tiles (lenstool-hpc_b200/csrc/lt_tree64.cu)
against the batch of the same request, whose tiles evaluate every halo at every pixel, and against
extended precision.  The bound is the batch's own (conftest.plane_close): 1e-13 of max(|ref|, RMS);
truncation (5e-15 of a far term) and the sums' rounding (n u of the sum of n = 450 terms of one
sign, 5e-14) stay below it."""
import numpy as np
import pytest

import lenstool_hpc_b200 as lt
from lenstool_hpc_b200 import catalog

from conftest import max_rel_err
from test_closed64 import _reference

pytestmark = pytest.mark.gpu
TOL = 1e-13


@pytest.fixture(scope="module")
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    c = lt.Context(0)
    yield c
    c.close()


def _catalog(n, types, seed=3, spread=90., e=0.5, clusters=2):
    rng = np.random.default_rng(seed)
    base = catalog.cluster_galaxy_parameters(clusters, n - clusters, seed)
    pos = rng.uniform(-spread, spread, (2, n))
    return catalog.make_catalog(rng.choice(np.array(types, np.int32), n), pos[0], pos[1], base.vdisp,
                                np.minimum(base.ellipticity * e / 0.5, 0.95), base.ellipticity_angle, base.rcore,
                                base.rcut, dlsds=rng.choice([0.5, 0.8], n))


def _dev(g):
    import torch
    return torch.full((g.ny, g.nx), np.nan, dtype=torch.float64, device="cuda")


def _direct(ctx, cat, g, kinds, scale):
    """Deflection and potential of every pair: the batch's tiles."""
    out = {k: _dev(g) for k in kinds}
    h = ctx.upload(cat)
    b = ctx.batch([lt.Request(h, g, out, scale=scale)], precision="fp64")
    b.launch()
    ctx.synchronize()
    b.destroy()
    return {k: v.cpu().numpy() for k, v in out.items()}


GRIDS = {
    "ordinary": catalog.Grid.square(100., 640),
    "odd": catalog.Grid(-100., 80., -70., 95., 701, 523),
    "thin": catalog.Grid(-90., 90., -1., 1., 1600, 33),
    "falling": catalog.Grid(100., -100., 60., -90., 600, 450, dx=-200. / 599, dy=-150. / 449),
    "offset": catalog.Grid(-200., 200., -150., 150., 617, 401, 333, 250, dx=0.21, dy=0.34),
    "cut-out": catalog.Grid(5., 35., -40., -10., 512, 512),
    "small": catalog.Grid.square(100., 250),
    "one parent wide": catalog.Grid(-3., 3., -90., 90., 50, 3000),
}


@pytest.mark.parametrize("types", [[81], [8, 81], [5, 8, 81, 81]])
@pytest.mark.parametrize("grid", sorted(GRIDS))
def test_equals_the_direct_sums(ctx, grid, types):
    g = GRIDS[grid]
    cat = _catalog(450, types)
    want = _direct(ctx, cat, g, ["deflection_x", "deflection_y", "potential"], 0.7)
    for precision in ("fp64", "fp64fast"):
        ax, ay, psi = _dev(g), _dev(g), _dev(g)
        ctx.gradient_grid(cat, g, precision=precision, scale=0.7, out=(ax, ay))
        ctx.potential_grid(cat, g, precision=precision, scale=0.7, out=psi)
        ctx.synchronize()
        for got, k in ((ax, "deflection_x"), (ay, "deflection_y"), (psi, "potential")):
            assert max_rel_err(got.cpu().numpy(), want[k]) <= TOL, (precision, k)
        # host outputs, computed in bands of rows: the same planes
        hx, hy = ctx.gradient_grid(cat, g, precision=precision, scale=0.7)
        assert np.array_equal(hx, ax.cpu().numpy()) and np.array_equal(hy, ay.cpu().numpy())
        assert np.array_equal(ctx.potential_grid(cat, g, precision=precision, scale=0.7), psi.cpu().numpy())


@pytest.mark.parametrize("e", [0.02, 0.5, 0.95])
@pytest.mark.parametrize("kmap", [False, True])
def test_fast_lens_maps_against_extended_precision(ctx, e, kmap):
    """Convergence and shear (weighted for the Kmap) and the potential at seeded pixels."""
    cat = _catalog(300, [8, 81, 81], seed=8, e=e)
    g = catalog.Grid(-100., 100., -80., 80., 901, 655)
    idx = np.random.default_rng(1).choice(g.npix, 800, replace=False)
    px, py = g.coords(idx)
    ref = [np.zeros(idx.size, np.longdouble) for _ in range(4)]
    for i in range(cat.n):
        _, _, p, k, g1, g2 = _reference(int(cat.type[i]), cat.ellipticity_potential[i], cat.b0[i], cat.rcore[i],
                                        cat.rcut[i], cat.ellipticity_angle[i], px - np.longdouble(cat.position_x[i]),
                                        py - np.longdouble(cat.position_y[i]))
        w = cat.dlsds[i] if kmap else 1.
        for r, t in zip(ref, (w * k, w * g1, w * g2, p)):
            r += t
    m = ctx.hessian_maps(cat, g, ["kappa", "gamma1", "gamma2"], precision="fp64fast", kmap=kmap)
    for k, r in zip(("kappa", "gamma1", "gamma2"), ref):
        assert max_rel_err(m[k].ravel()[idx], r) <= TOL, k
    if not kmap:
        out = ctx.lens_maps(cat, g, precision="fp64fast", which=("kappa", "gamma1", "gamma2", "psi"))
        for k, r in zip(("kappa", "gamma1", "gamma2", "psi"), ref):
            assert max_rel_err(out[k].ravel()[idx], r) <= TOL, k
        assert max_rel_err(ctx.lens_maps(cat, g, precision="fp64", which=("psi",))["psi"].ravel()[idx], ref[3]) <= TOL


@pytest.mark.parametrize("rcore", [0.1, 15., 60.])
def test_halo_centre_on_a_pixel(ctx, rcore):
    """The potential is 0/0 at a centre, in a core wider than the tile too: NaN where the batch has it."""
    n = 200
    rng = np.random.default_rng(5)
    cat = catalog.make_catalog([81] * n, np.r_[0., 25., rng.uniform(-90., 90., n - 2)],
                               np.r_[0., -50., rng.uniform(-90., 90., n - 2)], rng.uniform(80., 300., n),
                               rng.uniform(0.05, 0.5, n), rng.uniform(0., np.pi, n), np.r_[rcore, rcore, np.full(n - 2, 0.1)],
                               np.full(n, 200.))
    g = catalog.Grid(-100., 100., -100., 100., 641, 641)  # steps of 0.3125
    want = _direct(ctx, cat, g, ["deflection_x", "deflection_y", "potential"], 1.0)
    ax, ay, psi = _dev(g), _dev(g), _dev(g)
    ctx.gradient_grid(cat, g, out=(ax, ay))
    ctx.potential_grid(cat, g, out=psi)
    ctx.synchronize()
    for got, k in ((ax, "deflection_x"), (ay, "deflection_y"), (psi, "potential")):
        got, ok = got.cpu().numpy(), np.isfinite(want[k])
        assert np.array_equal(np.isfinite(got), ok), k
        assert max_rel_err(np.where(ok, got, 0.), np.where(ok, want[k], 0.)) <= TOL, k
    assert np.isnan(want["potential"][320, 320])


@pytest.mark.parametrize("n", [129, 2049, 4000])
def test_many_near_halos(ctx, n):
    """Halos crowded into one tile: more of them near than are staged at once (128), and more
    than a tile's list holds (2048: that tile evaluates every halo at every pixel)."""
    cat = _catalog(n, [81], spread=2., clusters=0)
    far = _catalog(500, [5, 81], seed=11, clusters=0)
    both = catalog.HaloCatalog(**{f: np.concatenate([getattr(cat, f), getattr(far, f)]) for f in ("type",) + catalog.FIELDS})
    cat = both.sorted_by_type()
    g = catalog.Grid.square(100., 1024)
    want = _direct(ctx, cat, g, ["deflection_x", "deflection_y"], 1.0)
    ax, ay = _dev(g), _dev(g)
    ctx.gradient_grid(cat, g, out=(ax, ay))
    ctx.synchronize()
    assert max_rel_err(ax.cpu().numpy(), want["deflection_x"]) <= TOL * max(1., n / 450)
    assert max_rel_err(ay.cpu().numpy(), want["deflection_y"]) <= TOL * max(1., n / 450)


def test_captured(ctx):
    """A call in a stream capture allocates nothing and replays."""
    import torch
    cat = ctx.upload(_catalog(450, [81]))
    g = GRIDS["ordinary"]
    a, b = (_dev(g), _dev(g)), (_dev(g), _dev(g))
    s = torch.cuda.Stream()
    ctx.gradient_grid(cat, g, out=a, stream=s)
    s.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        ctx.gradient_grid(cat, g, out=b, stream=s)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
