"""The FP64 product where one displacement component is far larger than what the
others' forces come from: rigid translations, fields whose modes do not couple,
and magnitudes at the lower end of FP64's range.  What the large component must
not contribute is left out of the reference, so its bound is the operator
tests', relative to the small forces."""
import numpy as np
import pytest

from v119_2025_12_19_hexatop_aws_gb300 import _lib
from v119_2025_12_19_hexatop_aws_gb300.solver import apply_operator

pytestmark = pytest.mark.gpu

DIMS = (33, 12, 7)


def product(ctx, oracle, fac, u, nu=0.3, h=(1.0, 1.0, 1.0)):
    g = oracle.Grid(*DIMS, *h)
    ref = oracle.apply_A(g, oracle.canonical_stiffness(*h, nu), fac, u.reshape(-1), np.zeros(g.ndof, bool))
    y = apply_operator(_lib.make_grid(*DIMS, *h), fac, u.reshape(-1), nu=nu, ctx=ctx)
    return y.reshape(-1, 3), ref.reshape(-1, 3)


def factors(rng, contrast):
    n = DIMS[0] * DIMS[1] * DIMS[2]
    return 1e-9 + rng.uniform(0.0, 1.0, n) ** 3 if contrast else np.ones(n)


def noise(rng, *scale):
    return rng.standard_normal((DIMS[2] + 1, DIMS[1] + 1, DIMS[0] + 1, 3)) * scale


@pytest.mark.parametrize("contrast", [False, True])
@pytest.mark.parametrize("big", [0, 1, 2])
@pytest.mark.parametrize("eps", [1.0, 1e-3, 1e-6, 1e-12])
def test_translation_of_one_component(ctx, oracle, rng, contrast, big, eps):
    fac = factors(rng, contrast)
    u = noise(rng, eps, eps, eps)
    u[..., big] = 0.0
    _, ref = product(ctx, oracle, fac, u)
    u[..., big] = -1.7
    y, _ = product(ctx, oracle, fac, u)
    assert (np.abs(y - ref).max(0) <= 1e-13 * np.abs(ref).max(0)).all()


@pytest.mark.parametrize("contrast", [False, True])
@pytest.mark.parametrize("nu,h", [(0.3, (1.0, 1.0, 1.0)), (0.45, (1.0, 1.0, 1.0)), (0.3, (1.0, 1.0, 0.5))])
@pytest.mark.parametrize("eps", [1e-1, 1e-3, 1e-6, 1e-12])
def test_modes_that_do_not_couple(ctx, oracle, rng, contrast, nu, h, eps):
    """u_z as a function of y does not reach forces in x; alternating in all three directions, in x or y."""
    fac = factors(rng, contrast)
    u = noise(rng, eps, eps, 0.0)
    _, ref = product(ctx, oracle, fac, u, nu, h)
    u[..., 2] = rng.standard_normal(DIMS[1] + 1)[None, :, None]
    y, _ = product(ctx, oracle, fac, u, nu, h)
    assert np.abs(y - ref)[:, 0].max() <= 1e-13 * np.abs(ref[:, 0]).max()
    s = [np.where(np.arange(n + 1) % 2, -1.0, 1.0) for n in DIMS[::-1]]
    u[..., 2] = s[0][:, None, None] * s[1][None, :, None] * s[2][None, None, :]
    y, _ = product(ctx, oracle, fac, u, nu, h)
    assert (np.abs(y - ref)[:, :2].max(0) <= 1e-13 * np.abs(ref[:, :2]).max(0)).all()


@pytest.mark.parametrize("scale", [1e-305, 1e-300, 1e-290, 1e300])
def test_magnitudes_at_the_ends_of_the_range(ctx, oracle, rng, scale):
    fac = factors(rng, False)
    u = noise(rng, 1.0, 1.0, 1.0)
    _, ref = product(ctx, oracle, fac, u)
    y, _ = product(ctx, oracle, fac, u * scale)
    # values below 2^-1022 / 2^-53 = 2e-292 times their largest lose bits to the range itself
    assert np.abs(y / scale - ref).max() <= max(1e-13, 1e-323 / scale * 24) * np.abs(ref).max()


def test_subnormal_displacements(ctx, oracle, rng):
    fac = factors(rng, False)
    u = np.rint(noise(rng, 1.0, 1.0, 1.0) * 1e6)
    _, ref = product(ctx, oracle, fac, u)
    y, _ = product(ctx, oracle, fac, u * 2.0 ** -1074)
    # sums of up to 8 elements, each rounded to the spacing 2^-1074
    assert np.abs(y * 2.0 ** 1000 * 2.0 ** 74 - ref).max() <= 8.0


@pytest.mark.parametrize("contrast", [False, True])
@pytest.mark.parametrize("eps", [1e-3, 1e-8, 1e-10, 1e-13])
def test_small_strains_on_a_large_translation(ctx, oracle, rng, contrast, eps):
    fac = factors(rng, contrast)
    u = noise(rng, eps, eps, eps) - 1.7
    _, ref = product(ctx, oracle, fac, u + 1.7)  # exact: values within a factor of two of 1.7
    y, _ = product(ctx, oracle, fac, u)
    assert np.abs(y - ref).max() <= 1e-13 * np.abs(ref).max()
