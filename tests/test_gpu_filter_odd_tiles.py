"""The filter on cross-sections whose tile is 53 x 5 or 5 x 53 nodes (385 with
its halo, one past a multiple of 64), against the reference's loop."""
import numpy as np
import pytest

from v119_2025_12_19_hexatop_aws_gb300 import _lib
from v119_2025_12_19_hexatop_aws_gb300.helmholtz import filter_density

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(52, 4, 7), (4, 52, 7), (105, 4, 3), (104, 4, 20), (4, 105, 2)])
def test_filter_on_tiles_of_an_odd_node_count(ctx, oracle, rng, dims):
    g = oracle.Grid(*dims)
    rho = rng.uniform(0, 1, g.nelem)
    ref, it, _ = oracle.helmholtz_reference(g, rho, 0.9, tol=1e-9, max_iter=200, quirk=True)
    grid = _lib.make_grid(*dims)
    out, st = filter_density(grid, rho, 0.9, tol=1e-9, quirk=True, ctx=ctx)
    # the same PCG in another order of summation: the filter tests' bounds
    assert st["iterations"] == it
    assert np.abs(out - ref).max() <= 1e-10
    o32, _ = filter_density(grid, rho, 0.9, tol=1e-6, quirk=True, precision="fp32", ctx=ctx)
    assert np.abs(o32 - ref).max() <= 1e-5
