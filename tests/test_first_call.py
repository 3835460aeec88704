"""A process's first call, on a stream that does not wait for the default one: the interpolation tables uploaded by
lt_create are in place."""
import pathlib
import subprocess
import sys

import pytest

CODE = """
import sys
sys.path.insert(0, %r)
from conftest import load_package
lt = load_package()
import torch
from lenstool_hpc_b200 import catalog
s = torch.cuda.Stream()
g = catalog.Grid.square(100., 640)
a, b = (tuple(torch.empty((g.ny, g.nx), dtype=torch.float64, device="cuda") for _ in range(2)) for _ in range(2))
torch.cuda.synchronize()
cat = catalog.cluster_galaxy_catalog(2, 298, 1)
ctx = lt.Context(0)
ctx.gradient_grid(cat, g, out=a, stream=s)
s.synchronize()
ctx.gradient_grid(cat, g, out=b)
ctx.synchronize()
assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1]) and bool(a[0].abs().max() > 1.)
"""


@pytest.mark.gpu
def test_first_call_on_a_non_blocking_stream():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    here = str(pathlib.Path(__file__).resolve().parent)
    r = subprocess.run([sys.executable, "-c", CODE % here], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
