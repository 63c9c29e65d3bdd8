"""Kernels that march through element layers in chunks picked by the grid's size:
each element's values are the same in a slab of the grid, whose chunks differ."""
import ctypes as C

import numpy as np
import pytest
import torch

from v119_2025_12_19_hexatop_aws_gb300 import _lib
from v119_2025_12_19_hexatop_aws_gb300.topopt import sensitivities

pytestmark = pytest.mark.gpu

# one-layer chunks, a few layers, the longest
DIMS = [(33, 5, 17), (96, 47, 49), (250, 121, 83)]


def fields(rng, dims):
    nx, ny, nz = dims
    return rng.uniform(0.01, 1.0, (nz, ny * nx)), rng.standard_normal((nz + 1, 3 * (ny + 1) * (nx + 1)))


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("penal", [3.0, 2.5])
def test_sensitivities_of_a_slab(ctx, rng, dims, penal):
    nx, ny, nz = dims
    rho, u = fields(rng, dims)
    dc, _ = sensitivities(_lib.make_grid(*dims), rho.reshape(-1), u.reshape(-1), penal=penal, ctx=ctx)
    dc = dc.reshape(nz, -1)
    for k0, k1 in [(0, 1), (nz - 3, nz), (5, 12)]:
        part, _ = sensitivities(_lib.make_grid(nx, ny, k1 - k0), rho[k0:k1].reshape(-1),
                                np.ascontiguousarray(u[k0:k1 + 1]).reshape(-1), penal=penal, ctx=ctx)
        assert np.array_equal(part.reshape(k1 - k0, -1), dc[k0:k1])


@pytest.mark.parametrize("dims", DIMS)
def test_stresses_of_a_slab(ctx, rng, dims):
    nx, ny, nz = dims
    rho, u = fields(rng, dims)

    def stress(k0, k1):
        ne = nx * ny * (k1 - k0)
        d = torch.from_numpy(rho[k0:k1].astype(np.float32)).cuda()
        x = torch.from_numpy(u[k0:k1 + 1]).cuda()
        out = [torch.empty(m * ne, device="cuda") for m in (3, 1, 6, 1, 3, 3)]
        torch.cuda.synchronize()  # the context works on a stream of its own
        grid = _lib.make_grid(nx, ny, k1 - k0)
        ctx.check(ctx.lib.hexa_stress_field(ctx.h, C.byref(grid), _lib.ptr(x), _lib.ptr(d), 1.0, 0.3,
                                            *[_lib.ptr(a) for a in out]))
        return [a.cpu().numpy().reshape(k1 - k0, -1) for a in out]

    whole = stress(0, nz)
    for k0, k1 in [(0, 1), (nz - 3, nz), (5, 12)]:
        for a, b in zip(whole, stress(k0, k1)):
            assert np.array_equal(a[k0:k1], b)  # unit elements: the Jacobian is exact at any height
