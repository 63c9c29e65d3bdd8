"""The filter's tiled PCG where its tiles can go wrong: cross-sections one node
past a tile, single-element axes, several z-chunks, more items than CTAs, and
the output written over the input."""
import numpy as np
import pytest
import torch

from v119_2025_12_19_hexatop_aws_gb300 import _lib
from v119_2025_12_19_hexatop_aws_gb300.helmholtz import filter_density

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(64, 5, 2), (1, 299, 1), (36, 6, 67), (2, 2, 401), (257, 1, 5), (1, 20000, 1)])
@pytest.mark.parametrize("quirk", [True, False])
def test_filter_tiles_follow_the_reference_loop(ctx, oracle, rng, dims, quirk):
    g = oracle.Grid(*dims)
    rho = rng.uniform(0, 1, g.nelem)
    ref, it, res = oracle.helmholtz_reference(g, rho, 0.9, tol=1e-9, max_iter=200, quirk=quirk)
    grid = _lib.make_grid(*dims)
    out, st = filter_density(grid, rho, 0.9, tol=1e-9, quirk=quirk, ctx=ctx)
    # the same PCG in another order of summation: the filter tests' 1e-10
    assert st["iterations"] == it
    assert np.abs(out - ref).max() <= 1e-10
    dev = torch.from_numpy(rho).cuda()
    filter_density(grid, dev, 0.9, tol=1e-9, quirk=quirk, out=dev, ctx=ctx)
    assert np.array_equal(dev.cpu().numpy(), out)
    # FP32: the loop's tolerance plus FP32 rounding over the few dozen iterations
    o32, _ = filter_density(grid, rho, 0.9, tol=1e-6, quirk=quirk, precision="fp32", ctx=ctx)
    assert np.abs(o32 - ref).max() <= 1e-5
