"""SIMP factors and sensitivities over every form of the penalty (whole
penalties take products, others pow), grids around a tile and a z-chunk, bricks
and Poisson ratios."""
import numpy as np
import pytest

from v119_2025_12_19_hexatop_aws_gb300 import _lib
from v119_2025_12_19_hexatop_aws_gb300.topopt import sensitivities, simp_factors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("penal", [1.0, 2.0, 3.0, 4.0, 5.0, 6.0, 7.0, 1.5, 2.9999999])
def test_simp_factors(ctx, rng, penal):
    rho = np.concatenate([rng.uniform(0.0, 1.0, 1000), [0.0, 1.0, 1e-3, 1e-200, 1e200, np.inf, np.nan]])
    out = simp_factors(rho, 1e-9, 1.0, penal, ctx=ctx)
    with np.errstate(over="ignore", under="ignore"):
        ref = 1e-9 + (rho.astype(np.longdouble) ** np.longdouble(penal)) * (1 - np.longdouble(1e-9))
        ref = ref.astype(np.float64)
    assert np.array_equal(np.isnan(out), np.isnan(ref)) and np.array_equal(np.isinf(out), np.isinf(ref))
    ok = np.isfinite(ref)
    # the power to an ulp, a product and a sum: 2.5 ulp
    assert (np.abs(out - ref)[ok] <= 2.5 * 2.3e-16 * np.abs(ref[ok])).all()


@pytest.mark.parametrize("dims,h", [((1, 1, 1), (1, 1, 1)), ((33, 5, 17), (1, 1, 0.5)), ((31, 3, 33), (0.3, 2, 0.7)),
                                    ((64, 4, 16), (1, 1, 1))])
@pytest.mark.parametrize("nu", [0.0, 0.3, 0.45])
@pytest.mark.parametrize("penal", [3.0, 1.0, 2.5])
def test_sensitivities(ctx, oracle, rng, dims, h, nu, penal):
    g = oracle.Grid(*dims, *h)
    rho = rng.uniform(0.01, 1.0, g.nelem)
    u = rng.standard_normal(g.ndof)
    dc, c = sensitivities(_lib.make_grid(*dims, *h), rho, u, nu=nu, penal=penal, ctx=ctx)
    rdc, rc = oracle.sensitivities(g, oracle.canonical_stiffness(*h, nu), rho, u, 1e-9, 1.0, penal)
    assert np.abs(dc - rdc).max() <= 1e-12 * np.abs(rdc).max()  # the topology tests' bound
    assert abs(c - rc) <= 1e-12 * abs(rc)
