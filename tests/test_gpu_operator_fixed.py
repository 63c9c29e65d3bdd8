"""The FP64 operator's integer element product: tile edges of its CTAs, bricks
and Poisson ratios on both sides of its rule, magnitudes over FP64's range, zero
and rigid fields, values that differ by many orders within an element, and
non-finite entries."""
import numpy as np
import pytest

from v119_2025_12_19_hexatop_aws_gb300 import _lib
from v119_2025_12_19_hexatop_aws_gb300.solver import apply_operator

pytestmark = pytest.mark.gpu


def both(ctx, oracle, dims, h, nu, fac, x, faces=1):
    g = oracle.Grid(*dims, *h)
    fixed = oracle.fixed_mask(g, faces) if faces else np.zeros(g.ndof, bool)
    ref = oracle.apply_A(g, oracle.canonical_stiffness(*h, nu), fac, np.where(fixed, 0.0, x), fixed)
    return apply_operator(_lib.make_grid(*dims, *h), fac, x, nu=nu, clamp_faces=faces, ctx=ctx), ref


@pytest.mark.parametrize("dims", [(1, 1, 1), (31, 10, 2), (30, 11, 3), (61, 22, 1), (5, 23, 40)])
@pytest.mark.parametrize("h,nu", [((1, 1, 1), 0.3), ((1, 1, 0.5), 0.0), ((0.3, 1, 0.7), 0.45), ((1, 1, 1), 0.4999),
                                  ((1, 1, 0.01), 0.3)])
def test_products_match_the_oracle(ctx, oracle, rng, dims, h, nu):
    n = dims[0] * dims[1] * dims[2]
    fac = np.where(rng.uniform(size=n) < 0.3, 1e-9, rng.uniform(0.1, 1.0, n))
    x = rng.standard_normal(3 * (dims[0] + 1) * (dims[1] + 1) * (dims[2] + 1))
    y, ref = both(ctx, oracle, dims, h, nu, fac, x)
    assert np.abs(y - ref).max() <= 1e-13 * np.abs(ref).max()  # the operator tests' bound


@pytest.mark.parametrize("scale", [1e-250, 1e-100, 1.0, 1e100, 1e250])
def test_magnitudes(ctx, oracle, rng, scale):
    dims = (9, 12, 5)
    fac = rng.uniform(0.1, 1.0, 540)
    x = rng.standard_normal(3 * 10 * 13 * 6)
    y, ref = both(ctx, oracle, dims, (1, 1, 1), 0.3, fac, x * scale)
    assert np.abs(y - ref).max() <= 1e-13 * np.abs(ref).max()
    assert np.isfinite(y).all() and np.abs(y).max() > 0


def test_zero_and_rigid_fields(ctx, oracle, rng):
    dims = (9, 12, 5)
    fac = rng.uniform(0.1, 1.0, 540)
    n = 10 * 13 * 6
    y, _ = both(ctx, oracle, dims, (1, 1, 1), 0.3, fac, np.zeros(3 * n), faces=0)
    assert not y.any()
    y, _ = both(ctx, oracle, dims, (1, 1, 1), 0.3, fac, np.tile([1.7, -0.3, 1e6], n), faces=0)
    assert np.abs(y).max() <= 1e-13 * 1e6


def test_orders_of_magnitude_within_an_element(ctx, oracle, rng):
    dims = (9, 12, 5)
    fac = rng.uniform(0.1, 1.0, 540)
    x = rng.standard_normal(3 * 10 * 13 * 6) * 10.0 ** rng.uniform(-12, 8, 3 * 10 * 13 * 6)
    x[rng.uniform(size=x.size) < 0.2] = 0.0
    x[5], x[100] = 5e-324, -1e-310
    y, ref = both(ctx, oracle, dims, (1, 1, 1), 0.3, fac, x)
    # per node against the largest displacement of the elements around it: FP64's own rounding unit times 24 terms
    g = oracle.Grid(*dims)
    big = np.abs(x).reshape(6, 13, 10, 3).max(-1)
    for ax in range(3):
        p = np.pad(big, [(1, 1) if a == ax else (0, 0) for a in range(3)])
        big = np.maximum(np.maximum(np.take(p, range(0, p.shape[ax] - 2), ax), np.take(p, range(2, p.shape[ax]), ax)),
                         big)
    assert (np.abs(y - ref).reshape(6, 13, 10, 3).max(-1) <= 24 * 2.3e-16 * 8 * big + 1e-300).all()
    assert g.ndof == y.size


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_entries_spread_as_in_the_element_product(ctx, oracle, rng, bad):
    dims = (9, 12, 5)
    fac = rng.uniform(0.1, 1.0, 540)
    x = rng.standard_normal(3 * 10 * 13 * 6)
    at = 3 * (4 + 10 * (6 + 13 * 2)) + 1
    x[at] = bad
    y, ref = both(ctx, oracle, dims, (1, 1, 1), 0.3, fac, x, faces=0)
    assert np.array_equal(np.isfinite(y), np.isfinite(ref))
    ok = np.isfinite(ref)
    assert np.abs(y[ok] - ref[ok]).max() <= 1e-13 * np.abs(ref[ok]).max()
