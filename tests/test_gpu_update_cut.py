"""The density update's selection where its shortcuts meet: the cut inside a
short list of ties, at its limit (1024) and beyond, exactly at the end of the
ties, and device arrays that a NaN stress must leave alone."""
import numpy as np
import pytest
import torch

from v119_2025_12_19_hexatop_aws_gb300 import _lib
from v119_2025_12_19_hexatop_aws_gb300.topopt import density_update_params, update_density_gpu

pytestmark = pytest.mark.gpu
F32 = np.float32


@pytest.mark.parametrize("ties", [1, 2, 700, 1024, 1025, 3000])
@pytest.mark.parametrize("cut", ["first", "inside", "last"])
def test_cut_among_equal_densities(ctx, rng, ties, cut):
    dims = (32, 20, 20)
    ne = 12800
    rho = rng.uniform(0.2, 0.9, ne).astype(F32)
    at = rng.permutation(ne)
    rho[at[:500]] = rng.uniform(0.05, 0.09, 500).astype(F32)
    rho[at[500:500 + ties]] = F32(0.1)
    k = 500 + {"first": 1, "inside": (ties + 1) // 2, "last": ties}[cut]
    ratio = F32((k + 0.5) / ne)  # floor(12800 * ratio) = k
    p = density_update_params(E=1.0, l1_stress_allowable=1.0, iter=30, number_of_iterations=30,
                              minimum_filter_radius_as_elements=0.0, max_culling_ratio=float(ratio),
                              max_domain_dim=1.0)
    orig = np.ones(ne, F32)
    d = np.ones(ne, F32)
    st = update_density_gpu(_lib.make_grid(*dims), d, rho, None, orig, p, ctx=ctx)
    ref = rho.copy()
    ref[np.argsort(rho, kind="stable")[:k]] = F32(1e-3)
    assert st["culled"] == k and st["active_count"] == ne
    assert np.array_equal(d, ref)
    dev = torch.ones(ne, device="cuda")
    torch.cuda.synchronize()  # the context works on a stream of its own
    update_density_gpu(_lib.make_grid(*dims), dev, torch.from_numpy(rho).cuda(), None, torch.from_numpy(orig).cuda(), p,
                       ctx=ctx)
    assert np.array_equal(dev.cpu().numpy(), ref)
    bad = torch.from_numpy(rho).cuda()
    bad[77] = float("nan")
    st = update_density_gpu(_lib.make_grid(*dims), dev, bad, None, torch.from_numpy(orig).cuda(), p, ctx=ctx)
    assert st["status"] == 1 and st["R_length"] == 0.0 and np.array_equal(dev.cpu().numpy(), ref)
