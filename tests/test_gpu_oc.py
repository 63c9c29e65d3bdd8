"""hexa_oc_update against the bisection evaluated multiplier by multiplier in
numpy: sizes around a block and a launch, entries with zero and positive
sensitivities, targets with no multiplier."""
import numpy as np
import pytest

from v119_2025_12_19_hexatop_aws_gb300.topopt import oc_update

pytestmark = pytest.mark.gpu


def bisection(x, dc, dv, volfrac, move):
    def new(lam):
        with np.errstate(invalid="ignore", divide="ignore"):
            be = x * np.sqrt(-dc / dv / lam)
        return np.fmax(0.0, np.fmax(x - move, np.fmin(1.0, np.fmin(x + move, be))))

    l1, l2, mid, levels = 0.0, 1e9, 5e8, 0
    while (l2 - l1) / (l1 + l2) > 1e-12 and levels < 320:
        mid = 0.5 * (l1 + l2)
        if new(mid).sum() > volfrac * x.size:
            l1 = mid
        else:
            l2 = mid
        levels += 1
    return new(mid), mid


@pytest.mark.parametrize("n", [1, 255, 257, 152 * 4 * 256 + 3])
@pytest.mark.parametrize("volfrac", [0.02, 0.3, 0.45, 0.99])
def test_oc_update_follows_the_bisection(ctx, n, volfrac):
    """0.02 and 0.99 lie outside what any multiplier reaches (x within 0.2 .. 0.8, move 0.15)."""
    rng = np.random.default_rng(n)
    x = rng.uniform(0.2, 0.8, n)
    dc = -np.exp(2.0 * rng.standard_normal(n) - 5.0)
    dv = rng.uniform(0.8, 1.2, n)
    if n > 1:
        dc[::17], dc[5::23] = 0.0, -dc[5::23]
    ref, lam = bisection(x, dc, dv, volfrac, 0.15)
    out, got = oc_update(x, dc, dv, volfrac, 0.15, ctx=ctx)
    # the bisection ends at a relative width of 1e-12
    assert got == pytest.approx(lam, rel=2e-12, abs=0.0)
    assert np.abs(out - ref).max() <= 2e-12
