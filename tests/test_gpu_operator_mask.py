"""The operator's masked reads: anything may stand at fixed DOFs of x (NaN
here), whichever way they are fixed; device and host masks; the result written
over its input."""
import ctypes as C

import numpy as np
import pytest
import torch

from v119_2025_12_19_hexatop_aws_gb300 import _lib
from v119_2025_12_19_hexatop_aws_gb300.solver import apply_operator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (30, 15, 3), (31, 14, 2), (33, 16, 5), (63, 8, 20)])
@pytest.mark.parametrize("faces", [0, 0b000001, 0b101010, 0b010101])
@pytest.mark.parametrize("dof_mask", [False, True])
@pytest.mark.parametrize("fp32", [False, True])
def test_operator_ignores_fixed_entries(ctx, oracle, rng, dims, faces, dof_mask, fp32):
    g = oracle.Grid(*dims)
    fac = rng.uniform(0.1, 1.0, g.nelem)
    x = rng.standard_normal(g.ndof)
    fixed = oracle.fixed_mask(g, faces) if faces else np.zeros(g.ndof, bool)
    fd = None
    if dof_mask:
        fd = (rng.uniform(size=g.ndof) < 0.1).astype(np.uint8) * 7
        fixed = fixed | (fd != 0)
    ref = oracle.apply_A(g, oracle.canonical_stiffness(1, 1, 1, 0.3), fac, np.where(fixed, 0.0, x), fixed)
    ref = ref + 0.25 * np.where(fixed, 0.0, x)
    bad = np.where(fixed, np.nan, x)
    dt = np.float32 if fp32 else np.float64
    grid = _lib.make_grid(*dims)
    y = apply_operator(grid, fac.astype(dt), bad.astype(dt), sigma=0.25, clamp_faces=faces, fixed_dof=fd, ctx=ctx,
                       fp32=fp32)
    tol = (2e-6 if fp32 else 1e-13) * max(np.abs(ref).max(), 1e-300)  # the operator tests' bounds
    assert np.abs(y - ref).max() <= tol
    assert not y[fixed].any()
    # device arrays, the mask on the device, y written over x
    xd, fcd = torch.from_numpy(bad.astype(dt)).cuda(), torch.from_numpy(fac.astype(dt)).cuda()
    md = None if fd is None else torch.from_numpy(fd).cuda()
    bc = _lib.make_bc(faces, md)
    fn = ctx.lib.hexa_apply_operator_f32 if fp32 else ctx.lib.hexa_apply_operator
    ctx.check(fn(ctx.h, C.byref(grid), C.byref(bc), 0.3, _lib.ptr(fcd), _lib.ptr(xd), 0.25, _lib.ptr(xd)))
    assert np.array_equal(xd.cpu().numpy(), y)
