"""The exact coarsest-level solve through one-level hierarchies, where the
V-cycle is the dense inverse itself: sizes around its 32-blocks and its limit
(2304 DOFs), clamped faces and a per-DOF mask, void contrast."""
import numpy as np
import pytest

from v119_2025_12_19_hexatop_aws_gb300 import _lib, workloads
from v119_2025_12_19_hexatop_aws_gb300.solver import solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(2, 2, 2), (3, 3, 1), (7, 6, 5), (12, 6, 6), (15, 7, 5), (16, 7, 5)])
@pytest.mark.parametrize("mask", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_one_level_multigrid_is_the_inverse(ctx, oracle, rng, dims, mask, precision):
    g = oracle.Grid(*dims)
    fac = rng.uniform(0.1, 1.0, g.nelem)
    fac[rng.uniform(size=g.nelem) < 0.2] = 1e-6
    fixed = oracle.fixed_mask(g, 1)
    if mask:
        fixed = fixed | (rng.uniform(size=g.ndof) < 0.03)
    f = workloads.edge_load(*dims)
    K0 = oracle.canonical_stiffness(1, 1, 1, 0.3)
    p = _lib.default_params(precision=precision, tol=1e-11, mg_levels=1, shift_factor=1e-10, coarse_iters=30)
    kw = {"fixed_dof": fixed.astype(np.uint8)} if mask else {"clamp_faces": 1}
    u, st = solve(_lib.make_grid(*dims), fac, f, params=p, ctx=ctx, **kw)
    ref = oracle.direct_solve(g, K0, fac, f, fixed, st["shift"])
    assert st["status"] == 0
    # u to the residual times a condition of about 1e4 (contrast 1e-6 behind a stiff frame)
    assert np.linalg.norm(u - ref) <= 1e-7 * np.linalg.norm(ref)
    if g.ndof <= 2304:
        # FP64: one application is the solution.  Mixed: FP32 rounding leaves a few steps per update.
        assert st["iterations"] <= (3 if precision == "fp64" else 40)
