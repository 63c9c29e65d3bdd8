"""The FP32 operator's dot product over items of several hundred layers: the step
length of the first Jacobi-PCG iteration on a grid whose z-chunks are the whole
of its height, for a direction whose terms are all alike (their rounding errors
add up instead of cancelling)."""
import pytest
import torch

from v119_2025_12_19_hexatop_aws_gb300 import _lib
from v119_2025_12_19_hexatop_aws_gb300.solver import apply_operator, solve

pytestmark = pytest.mark.gpu

U = 2.0 ** -24


@pytest.mark.parametrize("scale", [1.0, 1.13, 1.29, 1.47, 1.61, 1.87])
def test_step_length_on_long_items(ctx, scale):
    nx, ny, nz = 245, 283, 400  # 8 x 19 tiles of 31 x 15 nodes: one item of 401 layers for each SM
    grid = _lib.make_grid(nx, ny, nz)
    sign = [torch.ones(n + 1, device="cuda", dtype=torch.float64) for n in (nz, ny, nx)]
    for s in sign:
        s[1::2] = -1.0
    p = torch.empty((nz + 1, ny + 1, nx + 1, 3), device="cuda", dtype=torch.float64)
    p[..., 0] = scale * sign[2][None, None, :]
    p[..., 1] = scale * sign[1][None, :, None]
    p[..., 2] = scale * sign[0][:, None, None]
    count = [torch.full((n + 1,), 2.0, device="cuda", dtype=torch.float64) for n in (nz, ny, nx)]
    for c in count:
        c[0] = c[-1] = 1.0
    corner = torch.zeros(3 * 8, device="cuda", dtype=torch.float64)
    corner[0] = 1.0
    one = torch.ones(1, device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()  # the context works on a stream of its own
    dd = float(apply_operator(_lib.make_grid(1, 1, 1), one, corner, ctx=ctx)[0])
    diag = dd * count[0][:, None, None] * count[1][None, :, None] * count[2][None, None, :]
    b = (diag[..., None] * p).reshape(-1)
    fac = torch.ones(nx * ny * nz, device="cuda", dtype=torch.float64)
    u = torch.empty_like(b)
    torch.cuda.synchronize()
    params = _lib.default_params(precision="fp32", precond="jacobi", tol=1e-30, max_iter=1, shift_factor=0.0,
                                 max_shift_attempts=1, divergence_check=0, stagnation_tol=1e30)
    solve(grid, fac, b, params=params, u_out=u, ctx=ctx)
    Kp = apply_operator(grid, fac, p.reshape(-1), ctx=ctx)
    alpha = (b @ p.reshape(-1)) / (p.reshape(-1) @ Kp)
    got = (u @ p.reshape(-1)) / (p.reshape(-1) @ p.reshape(-1))
    # n equal terms summed in FP32: n U / 2.  p.Ap in 13 sums of 96 terms, r.z in sums of 32, and 20 roundings of
    # the diagonal, the direction, the element products and the step itself
    assert abs(float(got / alpha) - 1.0) <= (0.5 * (96 + 13 + 32) + 20) * U
