"""The delensing's FP32 pre-test (lenstool-hpc_b200/csrc/lt_chi2.cu) never changes an inclusion
test: predicted images equal to the oracle's FP64 tests on the same deflections, for sources all
over the field, efficiencies of both signs and zero, coarse grids whose cells fold over several
critical curves, and corners that are not finite."""
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


def _sources(frame, k, seed):
    rng = np.random.default_rng(seed)
    bx, by = rng.uniform(frame[0], frame[1], k), rng.uniform(frame[2], frame[3], k)
    bx[:k // 2] *= 0.1
    by[:k // 2] *= 0.1
    dr = rng.choice([0.6, 0.55, 0.9, 1., 0.2, 0., -0.5], k)
    return bx, by, dr


def _check(ctx, oracle_lib, cat, frame, n, bx, by, dr):
    h = ctx.upload(cat)
    ax, ay = ctx.gradient_grid(h, catalog.Grid(*frame, n, n))
    onf, ofx, ofy = oracle_lib.delense(n, frame, ax, ay, bx, by, dr)
    keep = np.flatnonzero(onf < lt.MAX_IMAGES)
    if keep.size == 0:
        return 0
    bx, by, dr = bx[keep], by[keep], dr[keep]
    nf, fx, fy = ctx.delense(h, frame, n, bx, by, dr)
    assert np.array_equal(nf, onf[keep])
    for i, k in enumerate(keep):
        assert np.array_equal(fx[i, :nf[i]], ofx[k, :nf[i]]) and np.array_equal(fy[i, :nf[i]], ofy[k, :nf[i]])
    return int(nf.sum())


@pytest.mark.parametrize("frame", [(-100., 100., -100., 100.), (-10., 30., -20., 15.), (4000., 4200., -900., -700.)])
@pytest.mark.parametrize("n", [2, 3, 9, 64, 257, 600])
def test_every_source_against_the_oracle(ctx, oracle_lib, frame, n):
    shift = (0.5 * (frame[0] + frame[1]), 0.5 * (frame[2] + frame[3]))
    cat = catalog.cluster_galaxy_catalog(2, 98, 5)
    cat.position_x = cat.position_x + shift[0]
    cat.position_y = cat.position_y + shift[1]
    bx, by, dr = _sources((frame[0] - shift[0], frame[1] - shift[0], frame[2] - shift[1], frame[3] - shift[1]), 60, n)
    found = sum(_check(ctx, oracle_lib, cat, frame, n, bx[s:s + k] + shift[0], by[s:s + k] + shift[1], dr[s:s + k])
                for s, k in ((0, 60), (0, 1), (7, 13)))
    assert n < 64 or found > 0


def test_a_corner_that_is_not_finite(ctx, oracle_lib):
    """A grid point on a SIS centre: its deflection is 0/0, and the reference's test takes every
    source to be inside the cells around it."""
    cat = catalog.make_catalog([5, 81], [0., 30.], [0., 5.], [300., 150.], [0.2, 0.3], [0.3, 1.], [0., 0.1], [0., 20.])
    rng = np.random.default_rng(2)
    assert _check(ctx, oracle_lib, cat, (-40., 40., -40., 40.), 81, rng.uniform(-30., 30., 20), rng.uniform(-30., 30., 20),
                  np.full(20, 0.7)) > 0


def test_the_kept_workspace_is_given_back(oracle_lib):
    """chi2 keeps its device workspace; a later allocation that the HBM budget would refuse takes
    it back instead."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    n = 256
    c = lt.Context(0, budget_bytes=2 * 8 * n * n + 600_000)
    cat = catalog.cluster_galaxy_catalog(2, 48, 5)
    frame = (-50., 50., -50., 50.)
    bx, by, dr = np.zeros(3), np.zeros(3), np.full(3, 0.6)
    h = c.upload(cat)
    first = c.delense(h, frame, n, bx, by, dr)
    big = c.upload(catalog.cluster_galaxy_catalog(2, 998, 5))  # needs more than the budget has left beside it
    again = c.delense(h, frame, 128, bx, by, dr)
    assert again[0].size == 3
    big.release()
    for a, b in zip(first, c.delense(h, frame, n, bx, by, dr)):
        assert np.array_equal(a, b)
    c.close()
