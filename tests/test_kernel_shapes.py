"""The kernel shape that a caller sets is the one that runs, on small grids too (read from a captured call's graph),
and lt_autotune's time is that of the call."""
import re

import pytest

import lenstool_hpc_b200 as lt
from lenstool_hpc_b200 import catalog

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ctx():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    c = lt.Context(0)
    yield c
    c.close()


def _kernels(call, path):
    """The kernels of a call on the stream it is given, by their mangled names."""
    import torch
    s = torch.cuda.Stream()
    call(s)
    s.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    graph.enable_debug_mode()
    with torch.cuda.graph(graph, stream=s):
        call(s)
    graph.debug_dump(str(path))
    names = re.findall(r"grid(?:32c|64)_kernelI(?:Li\d+E|Lb\dE)+", path.read_text())
    return {re.sub(r"L[ib](\d+)E", r"\1,", n) for n in names}


@pytest.mark.parametrize("precision, config, kernel", [
    ("fp32c", (2, 2, 256, 64), "grid32c_kernelI2,2,256,2,1,"),
    ("fp32c", (2, 3, 128, 32), "grid32c_kernelI2,2,128,3,2,"),
    ("fp64", (2, 1, 256, 64), "grid64_kernelI8,2,0,1,256,1,"),
])
def test_a_set_shape_runs_on_a_small_grid(ctx, tmp_path, precision, config, kernel):
    import torch
    cat = ctx.upload(catalog.cluster_galaxy_catalog(1, 20, 3))
    g = catalog.Grid.square(100., 96)
    out = [torch.empty((g.ny, g.nx), dtype=torch.float64, device="cuda")]

    def call(s):
        ctx.hessian_maps(cat, g, ["kappa"], precision=precision, out=out, stream=s)

    assert kernel not in _kernels(call, tmp_path / "a")  # by default: CTAs of 64 threads
    ctx.set_kernel_config(precision, "hessian", *config)
    assert kernel in _kernels(call, tmp_path / "b")


def test_autotune_returns_the_time_of_the_call(ctx):
    """A deflection whose far halos are interpolated: 0.22 ms, the kernels that evaluate every pair 1.4 ms and more."""
    import torch
    cat = ctx.upload(catalog.cluster_galaxy_catalog(2, 198, 20261203))
    ms = ctx.autotune(cat, "fp64", "deflection", grid_n=1024)[2]
    g = catalog.Grid.square(100., 1024)
    out = tuple(torch.empty((g.ny, g.nx), dtype=torch.float64, device="cuda") for _ in range(2))
    a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    for k in range(13):
        if k == 3:
            a.record()
        ctx.gradient_grid(cat, g, out=out)
    b.record()
    torch.cuda.synchronize()
    assert ms <= 3. * a.elapsed_time(b) / 10, ms
