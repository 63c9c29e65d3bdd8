"""An OC volume target below what the move limits leave: found at once, and the
result is that of the bisection, which ends at its upper multiplier."""
import numpy as np
import pytest

from v119_2025_12_19_hexatop_aws_gb300.topopt import oc_update

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 300, 152 * 4 * 256 + 3])
def test_target_below_the_lower_limits(ctx, n):
    rng = np.random.default_rng(n)
    x = rng.uniform(0.5, 0.9, n)
    dc, dv = -rng.uniform(0.1, 1.0, n), np.ones(n)
    before = ctx.kernel_launches
    out, lam = oc_update(x, dc, dv, 0.2, 0.1, ctx=ctx)
    # one pass, one group of steps that return at once, the update
    assert ctx.kernel_launches - before <= 1 + 6 + 1
    assert lam == pytest.approx(1e9, rel=2e-12)
    assert np.array_equal(out, np.maximum(x - 0.1, 0.0))
