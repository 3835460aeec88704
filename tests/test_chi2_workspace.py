"""The chi2's workspace: it is kept from call to call up to a bound, and a batch of models asks for no more than one
model's buffers where memory is short."""
import numpy as np
import pytest

import lenstool_hpc_b200 as lt
from lenstool_hpc_b200 import catalog
from lenstool_hpc_b200.images import ImageSystems

pytestmark = pytest.mark.gpu
FRAME = (-100., 100., -100., 100.)
MB = 1 << 20


def _systems(n):
    rng = np.random.default_rng(n)
    return ImageSystems(np.ones(n, np.int32), rng.uniform(-90., 90., n), rng.uniform(-90., 90., n), np.full(n, 0.6))


def _models(n):
    rng = np.random.default_rng(0)
    return [catalog.make_catalog([81] * 3, rng.uniform(-50., 50., 3), rng.uniform(-50., 50., 3), [60., 70., 80.],
                                 [0.2] * 3, [0.3] * 3, [0.1] * 3, [20.] * 3) for _ in range(n)]


@pytest.fixture(autouse=True)
def _gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")


def test_many_models_under_a_small_budget():
    """64 models of 2000 systems: 78 MB of work and results (1.2 MB a model) beside 5 MB of planes and systems."""
    models, s = _models(64), _systems(2000)
    with lt.Context(0) as c:
        want = c.chi2([c.upload(m) for m in models], FRAME, 512, s)
    with lt.Context(0, 16 * MB) as c:
        got = c.chi2([c.upload(m) for m in models], FRAME, 512, s)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


@pytest.mark.parametrize("n, kept", [(2048, True), (8000, False)])  # planes of 67 MB and of 1 GB
def test_workspace_kept_is_bounded(n, kept):
    import torch
    with lt.Context(0) as c:
        m, s = c.upload(_models(1)[0]), _systems(5)
        first = c.chi2(m, FRAME, 64, s)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        a = c.chi2(m, FRAME, n, s)
        used = free - torch.cuda.mem_get_info()[0]
        assert (16 * n * n <= used + 4 * MB) if kept else used <= 16 * MB
        assert a == c.chi2(m, FRAME, n, s) and first == c.chi2(m, FRAME, 64, s)
