"""Per-DOF masks: one whose buffer cannot be had fails the call instead of
leaving the DOFs free, and one that fixes nothing costs a solve nothing."""
import ctypes as C

import numpy as np
import pytest
import torch

from v119_2025_12_19_hexatop_aws_gb300 import _lib, workloads
from v119_2025_12_19_hexatop_aws_gb300.solver import solve

pytestmark = pytest.mark.gpu


def test_product_without_room_for_its_mask_fails(built_lib):
    dims = (499, 499, 439)  # 110 M nodes: 330 MB of host mask to stage
    nn = 500 * 500 * 440
    grid = _lib.make_grid(*dims)
    x = torch.ones(3 * nn, device="cuda")
    y = torch.empty_like(x)
    fac = torch.ones(499 * 499 * 439, device="cuda")
    fixed = np.zeros(3 * nn, np.uint8)
    fixed[0] = 1
    fresh = _lib.Context(0)
    try:
        # the kernels are loaded and warm before the memory goes
        small = torch.ones(24, device="cuda")
        fresh.check(fresh.lib.hexa_apply_operator_f32(fresh.h, C.byref(_lib.make_grid(1, 1, 1)), None, 0.3,
                                                      _lib.ptr(small), _lib.ptr(small), 0.0, _lib.ptr(y)))
        torch.cuda.synchronize()
        free, _ = torch.cuda.mem_get_info()
        hog = torch.empty(free - (256 << 20), device="cuda", dtype=torch.uint8)
        bc = _lib.make_bc(0, fixed)
        rc = fresh.lib.hexa_apply_operator_f32(fresh.h, C.byref(grid), C.byref(bc), 0.3, _lib.ptr(fac), _lib.ptr(x), 0.0,
                                               _lib.ptr(y))
        del hog
        torch.cuda.empty_cache()
        assert rc == _lib.HEXA_ERR_NOMEM
    finally:
        fresh.close()


def test_mask_that_fixes_nothing(ctx, rng):
    dims = (16, 8, 8)
    fac = rng.uniform(0.1, 1.0, 1024)
    f = workloads.edge_load(*dims)
    got = []
    for fixed in (None, np.zeros(workloads.ndof(*dims), np.uint8)):
        p = _lib.default_params(precision="fp64", tol=1e-10, mg_levels=2)
        before = ctx.kernel_launches
        u, st = solve(_lib.make_grid(*dims), fac, f, clamp_faces=1, fixed_dof=fixed, params=p, ctx=ctx)
        got.append((u, st["iterations"], ctx.kernel_launches - before))
    assert np.array_equal(got[0][0], got[1][0]) and got[0][1] == got[1][1]
    assert got[1][2] == got[0][2] + 1  # the packing of the mask
