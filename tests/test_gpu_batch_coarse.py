"""The batch's one-CTA coarse solve at the edges of its register form (1024
nodes), through one-level hierarchies."""
import numpy as np
import pytest

from v119_2025_12_19_hexatop_aws_gb300 import _lib, workloads
from v119_2025_12_19_hexatop_aws_gb300.solver import solve, solve_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [[(1, 1, 1), (3, 2, 1)], [(15, 7, 7), (7, 7, 7)], [(16, 7, 7), (2, 2, 2)],
                                  [(31, 7, 3), (5, 5, 5), (31, 3, 7)]])
@pytest.mark.parametrize("faces", [1, 1 | 8])
def test_batch_one_level_matches_single_solves(ctx, rng, dims, faces):
    grids = [_lib.make_grid(*d) for d in dims]
    facs = [rng.uniform(0.1, 1.0, d[0] * d[1] * d[2]) for d in dims]
    forces = [workloads.edge_load(*d) + 1e-3 * rng.standard_normal(workloads.ndof(*d)) for d in dims]
    p = _lib.default_params(precision="mixed", tol=1e-11, divergence_check=0, mg_levels=1, max_iter=5000)
    U, stats, rc = solve_batch(grids, facs, forces, clamp_faces=faces, params=p, ctx=ctx)
    assert rc == _lib.HEXA_OK
    p64 = _lib.default_params(precision="fp64", precond="jacobi", divergence_check=0, tol=1e-12)
    for i, g in enumerate(grids):
        u, _ = solve(g, facs[i], forces[i], clamp_faces=faces, params=p64, ctx=ctx)
        # as the batch tests: residual 1e-11 times the condition of these factors
        assert np.linalg.norm(U[i] - u) <= 1e-8 * np.linalg.norm(u), i


# hierarchies that end on levels 0 to 3, in one launch past level 0: all small;
# one whose coarsest grid takes the shared-memory forms with it, one the global
@pytest.mark.parametrize("dims", [[(6, 4, 4), (16, 8, 8), (36, 18, 18), (72, 24, 24), (20, 10, 10)],
                                  [(26, 10, 10), (40, 16, 16), (18, 14, 14), (44, 18, 18)],
                                  [(50, 26, 26), (48, 24, 24), (88, 16, 16)]])
@pytest.mark.parametrize("faces", [1, 1 | 2])
def test_batch_coarse_solves_of_several_levels(ctx, rng, dims, faces):
    grids = [_lib.make_grid(*d) for d in dims]
    facs = [rng.uniform(0.1, 1.0, d[0] * d[1] * d[2]) for d in dims]
    forces = [workloads.edge_load(*d) + 1e-3 * rng.standard_normal(workloads.ndof(*d)) for d in dims]
    p = _lib.default_params(precision="mixed", tol=1e-11, divergence_check=0, max_iter=5000)
    U, stats, rc = solve_batch(grids, facs, forces, clamp_faces=faces, params=p, ctx=ctx)
    assert rc == _lib.HEXA_OK
    p64 = _lib.default_params(precision="fp64", precond="jacobi", divergence_check=0, tol=1e-12)
    for i, g in enumerate(grids):
        u, _ = solve(g, facs[i], forces[i], clamp_faces=faces, params=p64, ctx=ctx)
        # as the batch tests: residual 1e-11 times the condition of these factors
        assert np.linalg.norm(U[i] - u) <= 1e-8 * np.linalg.norm(u), i
