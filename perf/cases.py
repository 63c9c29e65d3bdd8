"""What this library is timed on: one pass of each entry point that a topology
optimisation calls, over the sizes that the repository's configurations, tests
and benchmark use (48x24x24 up to 384x192x192 hex8 elements).

A case is one call (or the two model calls around a solve) on inputs that live
where such a program keeps them: device arrays for everything that a loop
around `hexa_solve` hands from step to step, host arrays for the drop-in of the
reference's filter.  The kinds:

  apply    one operator product y = (K + sigma I) x, what every PCG iteration
           and every residual check is made of: FP64 (the default precision)
           and FP32, clamped faces or a per-DOF mask of fixed degrees of
           freedom, unit cubes or bricks
  filter   the Helmholtz density filter of a SIMP step (FP64, device arrays)
  dropin   `apply_gpu_filter`, the reference's own filter call: Float32 on host
           arrays
  model    the SIMP material model around a solve: element factors before it,
           sensitivities and compliance after it
  oc       the optimality-criteria update that ends a SIMP step
  stress   the stress post-processing of a solved displacement field
  update   the stress-ratio density update with culling (no filter in it)
  solve    a whole mixed-precision multigrid solve of a cantilever with SIMP
           void contrast
  batch    a whole batch of cantilevers of uneven sizes, as a parameter study
           runs them
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from v119_2025_12_19_hexatop_aws_gb300 import _lib
from v119_2025_12_19_hexatop_aws_gb300.helmholtz import apply_gpu_filter, filter_density
from v119_2025_12_19_hexatop_aws_gb300.solver import apply_operator, solve, solve_batch
from v119_2025_12_19_hexatop_aws_gb300.topopt import density_update_params

DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64, F32 = torch.float64, torch.float32
NU, EMIN, E0 = 0.3, 1e-9, 1.0
OK = (_lib.HEXA_OK,)
_CTX = None


def _ctx() -> _lib.Context:
    """The process's library context, as a program keeps one."""
    global _CTX
    if _CTX is None:
        _CTX = _lib.Context(0)
    return _CTX


# ------------------------------------------------------------------ the cases
def _apply(name, nx, ny, nz, bits, mask=False, sigma=0.0, dz=1.0):
    return {"name": name, "kind": "apply", "nx": nx, "ny": ny, "nz": nz, "bits": bits, "mask": mask, "sigma": sigma,
            "dz": dz}


def listed() -> list[dict]:
    return [
        # the smallest grid in use (the 10-iteration SIMP loop of the tests): latency and launches
        _apply("apply_f64_48", 48, 24, 24, 64),
        # the plain FP64 solve's product on the 12.8 M DOF cantilever
        _apply("apply_f64_256", 256, 128, 128, 64),
        # the FP32 product on the 43 M DOF cantilever, the largest grid
        _apply("apply_f32_384", 384, 192, 192, 32),
        # a part with its own supports: per-DOF mask, odd sizes, bricks, shifted system
        _apply("apply_f32_mask_190", 190, 93, 61, 32, mask=True, sigma=1e-6, dz=0.5),
        # the SIMP step's density filter, 1.5 elements wide
        {"name": "filter_f64_256", "kind": "filter", "nx": 256, "ny": 128, "nz": 128, "r_elems": 1.5, "tol": 1e-5,
         "quirk": True},
        # the reference's own filter call between its iterations, on the host's arrays
        {"name": "dropin_f32_95", "kind": "dropin", "nx": 95, "ny": 47, "nz": 61, "r_elems": 2.5, "tol": 1e-5},
        # the material model before and after each solve
        {"name": "model_256", "kind": "model", "nx": 256, "ny": 128, "nz": 128, "penal": 3.0},
        # the design update that ends each SIMP step
        {"name": "oc_256", "kind": "oc", "nx": 256, "ny": 128, "nz": 128, "volfrac": 0.3, "move": 0.2},
        # stresses of a solution, everything that the exporters and the update read
        {"name": "stress_256", "kind": "stress", "nx": 256, "ny": 128, "nz": 128, "voigt": True},
        # the reference's density update with culling by rank
        {"name": "update_256", "kind": "update", "nx": 256, "ny": 128, "nz": 128, "iter": 10, "hard": False},
        # one whole solve, the step that the benchmark times, at an eighth of its elements
        {"name": "solve_mixed_192", "kind": "solve", "nx": 192, "ny": 96, "nz": 96, "steps": 3},
        # a parameter study: eight cantilevers of the sizes that the batch benchmark draws
        {"name": "batch_8", "kind": "batch", "sizes": "96,40,64,24,80,16,56,32"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["apply", "apply", "apply", "apply", "filter", "dropin", "model", "oc", "stress", "update",
                       "solve", "batch"])
    if kind == "solve":
        m = rng.choice([8, 16])
        nx = m * rng.randint(64 // m, 160 // m)
        ny = m * max(1, round(nx * rng.uniform(0.35, 0.6) / m))
        nz = m * max(1, round(nx * rng.uniform(0.35, 0.6) / m))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "steps": rng.choice([2, 3])}
    if kind == "batch":
        n = rng.randint(3, 8)
        return {"kind": kind, "sizes": ",".join(str(8 * rng.randint(2, 11)) for _ in range(n))}
    hi = {"apply": 320, "dropin": 128}.get(kind, 256)
    nx = _log_int(rng, 32, hi)
    ny, nz = (max(5, int(round(nx * rng.uniform(0.3, 0.5)))) for _ in range(2))
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz}
    if kind == "apply":
        c["bits"] = rng.choice([32, 64])
        if c["bits"] == 64:
            c["nx"], c["ny"], c["nz"] = min(nx, 250), min(ny, 125), min(nz, 125)
        c["mask"] = rng.random() < 0.35
        c["sigma"] = rng.choice([0.0, 0.0, 1e-10, 1e-6])
        c["dz"] = rng.choice([1.0, 1.0, 0.5, 0.8])
    elif kind == "filter":
        c.update(r_elems=round(rng.uniform(1.2, 4.0), 2), tol=rng.choice([1e-5, 1e-8]), quirk=rng.random() < 0.5)
    elif kind == "dropin":
        c.update(r_elems=round(rng.uniform(1.2, 4.0), 2), tol=1e-5)
    elif kind == "model":
        c["penal"] = rng.choice([1.5, 2.0, 3.0, 3.0, 3.0, 4.0])
    elif kind == "oc":
        c.update(volfrac=round(rng.uniform(0.15, 0.6), 3), move=rng.choice([0.05, 0.1, 0.2]))
    elif kind == "stress":
        c["voigt"] = rng.random() < 0.6
    elif kind == "update":
        c.update(iter=rng.randint(2, 35), hard=rng.random() < 0.3)
    return c


# ----------------------------------------------------------------- the inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _blur(t, width):
    """Three box averages of odd width along each axis (edges replicated)."""
    for _ in range(3):
        for axis in (2, 3, 4):
            pad = [0, 0, 0, 0, 0, 0]
            pad[2 * (4 - axis)] = pad[2 * (4 - axis) + 1] = width // 2
            k = [1, 1, 1]
            k[axis - 2] = width
            t = torch.nn.functional.avg_pool3d(torch.nn.functional.pad(t, pad, mode="replicate"), k, stride=1)
    return t


def _density(nx, ny, nz, seed, lo=1e-3, width=5):
    """A SIMP density: a smoothed Gaussian field of mean about 0.3, clipped to [lo, 1]."""
    g = torch.randn((1, 1, nz, ny, nx), generator=_gen(seed), device=DEV, dtype=F32)
    g = _blur(g, width)
    g = (g - g.mean()) / g.std()
    return (0.3 + 0.25 * g).clamp_(lo, 1.0).reshape(-1).to(F64)


def _displacement(nx, ny, nz, seed, noise):
    """A bending field with long-wave ripples and node-scale noise, (NZ, NY, NX, 3) flattened."""
    gen = _gen(seed + 101)
    x, y, z = (torch.linspace(0, 1, n + 1, device=DEV, dtype=F64) for n in (nx, ny, nz))
    X, Y, Z = x[None, None, :], y[None, :, None], z[:, None, None]
    u = torch.empty((nz + 1, ny + 1, nx + 1, 3), device=DEV, dtype=F64)
    ph = torch.rand((3, 4), generator=gen, device=DEV, dtype=F64)
    for c in range(3):
        ripple = torch.sin(6.0 * X + 6.3 * ph[c, 0]) * torch.cos(4.0 * Y + 6.3 * ph[c, 1]) * torch.cos(
            4.0 * Z + 6.3 * ph[c, 2])
        bend = -X * X if c == 2 else 0.4 * X * (Z - 0.5 if c == 0 else Y - 0.5)
        u[..., c] = bend + 0.2 * ph[c, 3] * ripple
    u += noise * torch.randn(u.shape, generator=gen, device=DEV, dtype=F32)
    u[:, :, 0, :] = 0.0
    return u.reshape(-1)


def _fixed_dofs(nx, ny, nz, seed):
    """x = 0 clamped, y = 0 a symmetry plane, and a few supported nodes, one byte per DOF."""
    gen = _gen(seed + 202)
    f = torch.zeros((nz + 1, ny + 1, nx + 1, 3), device=DEV, dtype=torch.uint8)
    f[:, :, 0, :] = 1
    f[:, 0, :, 1] = 1
    f |= (torch.rand(f.shape, generator=gen, device=DEV) < 5e-4).to(torch.uint8)
    return f.reshape(-1)


def _edge_load(nx, ny, nz, seed):
    """Unit load in -z over the nodes of the x = max, z = 0 edge, unevenly spread."""
    w = 0.5 + torch.rand((ny + 1,), generator=_gen(seed + 303), device=DEV, dtype=F64)
    f = torch.zeros((nz + 1, ny + 1, nx + 1, 3), device=DEV, dtype=F64)
    f[0, :, nx, 2] = -w / w.sum()
    return f.reshape(-1)


def _part(nx, ny, nz, seed, width=5):
    """SIMP factors of a cantilever: void contrast 1.3e-7, solid where the load enters."""
    rho = _density(nx, ny, nz, seed, lo=5e-3, width=width).reshape(nz, ny, nx)
    rho[:2, :, -2:] = 1.0
    return EMIN + rho.reshape(-1) ** 3 * (E0 - EMIN)


def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _batch_dims(case):
    return [(int(s), int(s) // 2, int(s) // 2) for s in case["sizes"].split(",")]


def _inputs(case, seed) -> dict:
    kind = case["kind"]
    if kind == "batch":
        dims = _batch_dims(case)
        return {"factors": [_part(*d, seed + 7 * i, width=3) for i, d in enumerate(dims)],
                "forces": [_edge_load(*d, seed + 7 * i) for i, d in enumerate(dims)]}
    d = _dims(case)
    if kind == "apply":
        dt = F64 if case["bits"] == 64 else F32
        rho = _density(*d, seed)
        fac = (EMIN + rho ** 3 * (E0 - EMIN)).to(dt)
        x = _displacement(*d, seed, 0.3).to(dt)
        return {"fac": fac, "x": x, "fixed": _fixed_dofs(*d, seed) if case["mask"] else None}
    if kind == "filter":
        return {"rho": _density(*d, seed, width=3)}
    if kind == "dropin":
        return {"rho": _density(*d, seed, width=3).to(F32).cpu().numpy()}
    if kind == "model":
        return {"rho": _density(*d, seed), "u": _displacement(*d, seed, 1e-3)}
    if kind == "oc":
        rho = _density(*d, seed)
        e = torch.exp(1.5 * torch.randn(rho.shape, generator=_gen(seed + 404), device=DEV, dtype=F64) - 6.0)
        return {"x": rho, "dc": -3.0 * rho ** 2 * e, "dv": torch.ones_like(rho)}
    if kind == "stress":
        return {"u": _displacement(*d, seed, 1e-3), "rho": _density(*d, seed).to(F32)}
    if kind == "update":
        rho = _density(*d, seed).to(F32)
        gen = _gen(seed + 505)
        l1 = rho * torch.exp(0.8 * torch.randn(rho.shape, generator=gen, device=DEV, dtype=F32)) * 200.0
        return {"rho": rho, "l1": l1, "orig": torch.ones_like(rho)}
    return {"fac": _part(*d, seed), "f": _edge_load(*d, seed)}


def _solver_params(steps):
    # the benchmark's smoother, fixed (V(steps, steps) Chebyshev, no autotuner); the tolerance lies below the
    # benchmark's 1e-9, between that and the tests' 1e-13, where the displacements are settled to nine digits
    return _lib.default_params(precision="mixed", precond="multigrid", tol=2e-11, max_iter=20000, pre_smooth=steps,
                               post_smooth=steps, cheb_ratio=10, divergence_check=0, shift_factor=0.0)


def _update_params(case):
    return density_update_params(E=1.0, l1_stress_allowable=200.0, iter=int(case["iter"]), number_of_iterations=30,
                                 minimum_filter_radius_as_elements=0.0, hard_update=int(case["hard"]),
                                 max_culling_ratio=0.1, max_domain_dim=float(max(_dims(case))))


def prepare(case, seed) -> dict:
    ctx = _ctx()
    s = {"case": case, "kind": case["kind"], "ctx": ctx, **_inputs(case, seed)}
    kind = case["kind"]
    if kind == "batch":
        s["grids"] = [_lib.make_grid(*d) for d in _batch_dims(case)]
        s["out"] = [torch.empty_like(f) for f in s["forces"]]
        s["params"] = _solver_params(2)
        return s
    nx, ny, nz = _dims(case)
    s["grid"] = _lib.make_grid(nx, ny, nz, 1.0, 1.0, case.get("dz", 1.0))
    ne, nn = nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1)

    def new(n, dt=F64):
        return torch.empty(n, device=DEV, dtype=dt)

    if kind == "filter":
        s["out"] = new(ne)
    elif kind == "model":
        s["fac"], s["dc"] = new(ne), new(ne)
    elif kind == "oc":
        s["out"] = new(ne)
    elif kind == "stress":
        s["out"] = {"principal": new(3 * ne, F32), "vonmises": new(ne, F32),
                    "voigt": new(6 * ne, F32) if case["voigt"] else None, "l1": new(ne, F32),
                    "dir_max": new(3 * ne, F32), "dir_min": new(3 * ne, F32)}
    elif kind == "update":
        s["params"] = _update_params(case)
    elif kind == "solve":
        s["out"] = new(3 * nn)
        s["params"] = _solver_params(case["steps"])
    return s


# -------------------------------------------------------------------- the run
def run(s):
    kind, ctx = s["kind"], s["ctx"]
    case = s["case"]
    if kind == "batch":
        u, _, _ = solve_batch(s["grids"], s["factors"], s["forces"], clamp_faces=1, nu=NU, params=s["params"],
                              u_out=s["out"], ctx=ctx)
        return u
    grid = s["grid"]
    if kind == "apply":
        return apply_operator(grid, s["fac"], s["x"], nu=NU, sigma=case["sigma"], clamp_faces=0 if case["mask"] else 1,
                              fixed_dof=s["fixed"], ctx=ctx, fp32=case["bits"] == 32)
    if kind == "filter":
        return filter_density(grid, s["rho"], case["r_elems"] / 2.5, tol=case["tol"], max_iter=200,
                              quirk=case["quirk"], out=s["out"], ctx=ctx)[0]
    if kind == "dropin":
        return apply_gpu_filter(s["rho"], grid.nx, grid.ny, grid.nz, 1.0, 1.0, 1.0, case["r_elems"] / 2.5,
                                tol=case["tol"])[0]
    if kind == "model":
        c, p = C.c_double(), float(case["penal"])
        rho, fac, dc = s["rho"], s["fac"], s["dc"]
        ctx.check(ctx.lib.hexa_simp_factors(ctx.h, rho.numel(), _lib.ptr(rho), EMIN, E0, p, _lib.ptr(fac)), allow=OK)
        ctx.check(ctx.lib.hexa_sensitivities(ctx.h, C.byref(grid), NU, _lib.ptr(rho), _lib.ptr(s["u"]), EMIN, E0, p,
                                             _lib.ptr(dc), C.byref(c)), allow=OK)
        return {"factors": fac, "dc": dc, "compliance": c.value}
    if kind == "oc":
        lam = C.c_double()
        ctx.check(ctx.lib.hexa_oc_update(ctx.h, s["x"].numel(), _lib.ptr(s["x"]), _lib.ptr(s["dc"]), _lib.ptr(s["dv"]),
                                         float(case["volfrac"]), float(case["move"]), _lib.ptr(s["out"]),
                                         C.byref(lam)), allow=OK)
        return {"x": s["out"], "lambda": lam.value}
    if kind == "stress":
        o = s["out"]
        ctx.check(ctx.lib.hexa_stress_field(ctx.h, C.byref(grid), _lib.ptr(s["u"]), _lib.ptr(s["rho"]), E0, NU,
                                            *[_lib.ptr(o[k]) for k in ("principal", "vonmises", "voigt", "l1",
                                                                       "dir_max", "dir_min")]), allow=OK)
        return o
    if kind == "update":
        st = _lib.DensityUpdateStats()
        ctx.check(ctx.lib.hexa_update_density(ctx.h, C.byref(grid), _lib.ptr(s["rho"]), _lib.ptr(s["l1"]), None,
                                              _lib.ptr(s["orig"]), C.byref(s["params"]), C.byref(st)), allow=OK)
        return {"density": s["rho"], "mean_change": st.mean_change, "active": st.active_count,
                "candidates": st.candidates, "culled": st.culled}
    return solve(grid, s["fac"], s["f"], clamp_faces=1, params=s["params"], u_out=s["out"], ctx=ctx)[0]


def work(case) -> dict:
    """Every input read once and every output written once; the arithmetic of
    one element product (45 multiply-adds and 144 additions in the modal
    basis) where the path has products."""
    if case["kind"] == "batch":
        ne = sum(a * b * c for a, b, c in _batch_dims(case))
        nn = sum((a + 1) * (b + 1) * (c + 1) for a, b, c in _batch_dims(case))
        return {"bytes": 8 * ne + 48 * nn, "flops": 234 * ne}
    nx, ny, nz = _dims(case)
    ne, nn = nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1)
    kind = case["kind"]
    if kind == "apply":
        w = case["bits"] // 8
        return {"bytes": w * (6 * nn + ne) + (3 * nn if case["mask"] else 0), "flops": 234 * ne}
    if kind == "filter":
        return {"bytes": 16 * ne, "flops": 30 * nn}
    if kind == "dropin":
        return {"bytes": 8 * ne, "flops": 30 * nn}
    if kind == "model":
        return {"bytes": 24 * nn + 24 * ne, "flops": 200 * ne}
    if kind == "oc":
        return {"bytes": 32 * ne, "flops": 10 * ne}
    if kind == "stress":
        return {"bytes": 24 * nn + (72 if case["voigt"] else 48) * ne, "flops": 300 * ne}
    if kind == "update":
        return {"bytes": 16 * ne, "flops": 6 * ne}
    return {"bytes": 8 * ne + 48 * nn, "flops": 234 * ne}


# ------------------------------------------- what the calls return, in 64 bits
_CORNERS = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]


def _gauss(dx, dy, zlo, zhi):
    """(N, dN/dx, weight) at the 2x2x2 Gauss points of the brick [0,dx] x [0,dy] x [zlo,zhi]."""
    a = 1.0 / math.sqrt(3.0)
    L = (dx, dy, zhi - zlo)
    for p in ((i, j, k) for i in (-a, a) for j in (-a, a) for k in (-a, a)):
        N, G = np.empty(8), np.empty((8, 3))
        for m, cor in enumerate(_CORNERS):
            s = [2 * v - 1 for v in cor]
            t = [0.5 * (1 + s[q] * p[q]) for q in range(3)]
            N[m] = t[0] * t[1] * t[2]
            for q in range(3):
                G[m, q] = s[q] / L[q] * math.prod(t[r] for r in range(3) if r != q)
        yield N, G, L[0] * L[1] * L[2] / 8.0


def _stiffness(dz):
    """The 24x24 element matrix for E = 1."""
    f = 1.0 / ((1 + NU) * (1 - 2 * NU))
    D = np.zeros((6, 6))
    D[:3, :3] = NU * f
    D[[0, 1, 2], [0, 1, 2]] = (1 - NU) * f
    D[[3, 4, 5], [3, 4, 5]] = 0.5 * (1 - 2 * NU) * f
    K = np.zeros((24, 24))
    for _, G, w in _gauss(1.0, 1.0, 0.0, dz):
        B = np.zeros((6, 24))
        for m in range(8):
            gx, gy, gz = G[m]
            B[:, 3 * m:3 * m + 3] = [[gx, 0, 0], [0, gy, 0], [0, 0, gz], [gy, gx, 0], [0, gz, gy], [gz, 0, gx]]
        K += w * B.T @ D @ B
    return torch.from_numpy(K).to(DEV)


def _element_values(v, k0, k1):
    """Corner values of the element layers [k0, k1) of a nodal field (NZ, NY, NX, c): (layers, ny, nx, 8, c)."""
    ny, nx = v.shape[1] - 1, v.shape[2] - 1
    return torch.stack([v[k0 + c:k1 + c, b:b + ny, a:a + nx] for a, b, c in _CORNERS], dim=3)


def _matrix_product(K, fac, v):
    """sum_e f_e K u_e of a nodal field v (NZ, NY, NX, c) for an element matrix K (8c x 8c)."""
    nz, ny, nx, nc = v.shape[0] - 1, v.shape[1] - 1, v.shape[2] - 1, v.shape[3]
    y = torch.zeros_like(v)
    for k0 in range(0, nz, 16):
        k1 = min(nz, k0 + 16)
        w = _element_values(v, k0, k1).reshape(k1 - k0, ny, nx, 8 * nc) @ K
        if fac is not None:
            w *= fac[k0:k1, :, :, None]
        w = w.reshape(k1 - k0, ny, nx, 8, nc)
        for m, (a, b, c) in enumerate(_CORNERS):
            y[k0 + c:k1 + c, b:b + ny, a:a + nx] += w[:, :, :, m]
    return y


def _exact_apply(case, i):
    nx, ny, nz = _dims(case)
    x = i["x"].to(F64).reshape(nz + 1, ny + 1, nx + 1, 3).clone()
    if case["mask"]:
        free = (i["fixed"] == 0).reshape(x.shape)
    else:
        free = torch.ones_like(x, dtype=torch.bool)
        free[:, :, 0, :] = False
    x *= free
    y = _matrix_product(_stiffness(case["dz"]), i["fac"].to(F64).reshape(nz, ny, nx), x)
    return ((y + case["sigma"] * x) * free).reshape(-1)


def _exact_filter(case, rho, quirk):
    """The Jacobi-PCG of (R^2 K + M) psi = b, tested every 10 iterations, at most 200."""
    nx, ny, nz = _dims(case)
    R = case["r_elems"] / 2.5
    K = np.zeros((8, 8))
    for N, G, w in _gauss(1.0, 1.0, -0.5, 1.0 if quirk else 0.5):
        K += w * (R * R * G @ G.T + np.outer(N, N))
    A = torch.from_numpy(K).to(DEV)
    one = torch.ones((nz, ny, nx), device=DEV, dtype=F64)

    def gather(e, per_corner):
        out = torch.zeros((nz + 1, ny + 1, nx + 1), device=DEV, dtype=F64)
        for m, (a, b, c) in enumerate(_CORNERS):
            out[c:c + nz, b:b + ny, a:a + nx] += e * per_corner[m]
        return out

    b = gather(rho.reshape(nz, ny, nx), [0.125] * 8)
    dinv = 1.0 / gather(one, [float(K[m, m]) for m in range(8)])
    bnorm = b.norm()
    x, r = torch.zeros_like(b), b.clone()
    z = r * dinv
    p, rz = z.clone(), (r * z).sum()
    for it in range(1, 201):
        q = _matrix_product(A, None, p[..., None])[..., 0]
        alpha = rz / (p * q).sum()
        x += alpha * p
        r -= alpha * q
        if it % 10 == 0 and bool(r.norm() / bnorm < case["tol"]):
            break
        z = r * dinv
        rz_new = (r * z).sum()
        p = z + (rz_new / rz) * p
        rz = rz_new
    return (sum(x[c:c + nz, m:m + ny, a:a + nx] for a, m, c in _CORNERS) / 8.0).reshape(-1)


def _exact_model(case, i):
    nx, ny, nz = _dims(case)
    K, p, rho = _stiffness(1.0), case["penal"], i["rho"]
    v = i["u"].reshape(nz + 1, ny + 1, nx + 1, 3)
    ce = torch.empty((nz, ny, nx), device=DEV, dtype=F64)
    for k0 in range(0, nz, 16):
        k1 = min(nz, k0 + 16)
        ue = _element_values(v, k0, k1).reshape(k1 - k0, ny, nx, 24)
        ce[k0:k1] = ((ue @ K) * ue).sum(-1)
    ce = ce.reshape(-1)
    fac = EMIN + rho ** p * (E0 - EMIN)
    return {"factors": fac, "dc": -p * rho ** (p - 1) * (E0 - EMIN) * ce, "compliance": float((fac * ce).sum())}


def _exact_oc(case, i):
    x, move = i["x"], case["move"]
    t = x * torch.sqrt(-i["dc"] / i["dv"])
    lo, hi = (x - move).clamp(min=0.0), (x + move).clamp(max=1.0)

    def new(lam):
        return torch.maximum(lo, torch.minimum(hi, t / math.sqrt(lam)))

    l1, l2, target = 0.0, 1e9, case["volfrac"] * x.numel()
    mid = 0.5 * (l1 + l2)
    while (l2 - l1) / (l1 + l2) > 1e-12:
        mid = 0.5 * (l1 + l2)
        if float(new(mid).sum()) > target:
            l1 = mid
        else:
            l2 = mid
    return {"x": new(mid), "lambda": mid}


def _exact_stress(case, i):
    """Centre stresses of the Float32 displacements; eigenvalues by the trigonometric formula.  The directions have
    no unique value (their sign, and more where two stresses are equal)."""
    nx, ny, nz = _dims(case)
    v = i["u"].to(F32).to(F64).reshape(nz + 1, ny + 1, nx + 1, 3)
    f = E0 / ((1 + NU) * (1 - 2 * NU))
    rho = i["rho"].to(F64).reshape(nz, ny, nx)
    voigt = torch.empty((nz, ny, nx, 6), device=DEV, dtype=F64)
    sgn = torch.tensor([[2 * q - 1 for q in c] for c in _CORNERS], device=DEV, dtype=F64)
    for k0 in range(0, nz, 16):
        k1 = min(nz, k0 + 16)
        g = torch.einsum("zyxmc,md->zyxcd", _element_values(v, k0, k1), 0.25 * sgn)
        e = [g[..., q, q] for q in range(3)]
        tr = e[0] + e[1] + e[2]
        s = f * rho[k0:k1]
        for q in range(3):
            voigt[k0:k1, ..., q] = s * ((1 - 2 * NU) * e[q] + NU * tr)
        for q, (a, b) in enumerate(((0, 1), (1, 2), (0, 2))):
            voigt[k0:k1, ..., 3 + q] = s * (0.5 - NU) * (g[..., a, b] + g[..., b, a])
    voigt = voigt.reshape(-1, 6)
    xx, yy, zz, xy, yz, xz = voigt.unbind(1)
    m = (xx + yy + zz) / 3
    a, b, c = xx - m, yy - m, zz - m
    off = xy * xy + yz * yz + xz * xz
    p = torch.sqrt((a * a + b * b + c * c + 2 * off) / 6)
    det = a * (b * c - yz * yz) - xy * (xy * c - yz * xz) + xz * (xy * yz - b * xz)
    t = torch.acos((det / (2 * p ** 3).clamp(min=1e-300)).clamp(-1, 1)) / 3
    s1, s3 = m + 2 * p * torch.cos(t), m + 2 * p * torch.cos(t + 2 * math.pi / 3)
    principal = torch.stack([s1, 3 * m - s1 - s3, s3], dim=1)
    vm = torch.sqrt(0.5 * ((xx - yy) ** 2 + (yy - zz) ** 2 + (zz - xx) ** 2) + 3 * off)
    return {"principal": principal.reshape(-1), "vonmises": vm, "voigt": voigt.reshape(-1) if case["voigt"] else None,
            "l1": principal.abs().sum(1), "dir_max": None, "dir_min": None}


def _exact_update(case, i):
    """The update in the Float32 operations that define it (the density is a Float32 field)."""
    lo, hi, it = np.float32(1e-3), 1.0, case["iter"]
    raw = ((i["l1"] / 200.0) / 1.0).clamp(min=float(lo))
    new = raw.clamp(max=hi)
    change = float((new.to(F64) - i["rho"].to(F64)).abs().sum())
    live = new > float(lo)
    thr = np.float32(0.95) if it > 30 else np.float32(0.95) * (np.float32(it) / np.float32(30))
    cand = torch.nonzero(live & (new < float(thr))).reshape(-1)
    active = int(live.sum())
    allowed = int(math.floor(np.float32(active) * np.float32(0.1)))
    if cand.numel() > allowed:
        order = torch.sort(new[cand], stable=True).indices
        culled = cand[order[:allowed]]
    else:
        culled = cand
    new[culled] = float(lo)
    if case["hard"]:
        new = torch.where(new > float(lo), torch.ones_like(new), new)
    return {"density": new.to(F64), "mean_change": change / max(1, int((raw > float(lo)).sum())), "active": active,
            "candidates": int(cand.numel()), "culled": int(culled.numel())}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("solve", "batch"):  # a direct factorisation of these grids takes minutes
        return None
    i = _inputs(case, seed)
    if kind == "apply":
        return _exact_apply(case, i)
    if kind == "filter":
        return _exact_filter(case, i["rho"], case["quirk"])
    if kind == "dropin":
        return _exact_filter(case, torch.from_numpy(i["rho"]).to(DEV).to(F64), True)
    if kind == "model":
        return _exact_model(case, i)
    if kind == "oc":
        return _exact_oc(case, i)
    if kind == "stress":
        return _exact_stress(case, i)
    return _exact_update(case, i)
