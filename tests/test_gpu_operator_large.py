"""FP32 operator on a grid of which one vector exceeds L2 (its kernels prefetch
ahead of the march): the product against the FP64 operator, and a solve whose
smoother, residual and product are those kernels, by its FP64 residual."""
import pytest
import torch

from v119_2025_12_19_hexatop_aws_gb300 import _lib
from v119_2025_12_19_hexatop_aws_gb300.solver import apply_operator, solve

pytestmark = pytest.mark.gpu


# 130 MB a vector: no dimension a multiple of a tile or a chunk, and four grids of a V-cycle
@pytest.mark.parametrize("dims", [(217, 223, 221), (216, 224, 224)])
def test_large_fp32_operator(ctx, dims):
    grid = _lib.make_grid(*dims)
    nn, ne = (dims[0] + 1) * (dims[1] + 1) * (dims[2] + 1), dims[0] * dims[1] * dims[2]
    gen = torch.Generator(device="cuda").manual_seed(5)
    fac = torch.rand(ne, generator=gen, device="cuda", dtype=torch.float64) * 0.9 + 0.1
    x = torch.randn(3 * nn, generator=gen, device="cuda", dtype=torch.float64)
    fac, x = fac.float().double(), x.float().double()  # the same values in both types
    fac32, x32, u = fac.float(), x.float(), torch.empty_like(x)
    f = torch.zeros_like(x)
    f.view(-1, dims[0] + 1, 3)[:, -1, 1] = -1.0
    torch.cuda.synchronize()  # the context works on a stream of its own
    ref = apply_operator(grid, fac, x, clamp_faces=1, ctx=ctx)
    y = apply_operator(grid, fac32, x32, clamp_faces=1, ctx=ctx, fp32=True)
    assert (y.double() - ref).abs().max() <= 2e-6 * ref.abs().max()  # the operator tests' bound

    params = _lib.default_params(precision="mixed", precond="multigrid", tol=1e-6)
    _, st = solve(grid, fac, f, clamp_faces=1, params=params, u_out=u, ctx=ctx)
    r = f - apply_operator(grid, fac, u, sigma=st["shift"], clamp_faces=1, ctx=ctx)
    assert r.norm() <= 1.001e-6 * f.norm()
