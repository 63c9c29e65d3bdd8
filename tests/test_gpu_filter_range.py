"""The filter's scaling by powers of two at the lower end of FP64's range: a part
of the density just above the smallest normal number."""
import numpy as np
import pytest

from v119_2025_12_19_hexatop_aws_gb300 import _lib
from v119_2025_12_19_hexatop_aws_gb300.helmholtz import filter_density

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [0.0, 3e-308, 1e-307, 1e-305])
def test_filter_of_values_near_the_smallest_normal(ctx, oracle, rng, scale):
    dims = (24, 7, 6)
    g = oracle.Grid(*dims)
    rho = rng.uniform(0.5, 1.0, g.nelem).reshape(6, 7, 24)
    rho[:, :, 8:] *= scale
    rho = rho.reshape(-1)
    ref, it, _ = oracle.helmholtz_reference(g, rho, 0.9, tol=1e-9, max_iter=200, quirk=True)
    out, st = filter_density(_lib.make_grid(*dims), rho, 0.9, tol=1e-9, quirk=True, ctx=ctx)
    assert st["iterations"] == it
    assert np.abs(out - ref).max() <= 1e-10  # the filter tests' bound
