"""The work that is timed: passes through the package's public entry points, over the range of
problems this repository's configurations, tests and benchmark use.

A case names an operator (2D / 3D Poisson, upwind convection-diffusion, variable-coefficient
diffusion, a batch of 2D Poisson systems), a preconditioner with the type of its factor values,
and the call a program makes.  A program builds the operator, its DeviceSystem and its
preconditioner once and then calls with one right-hand side after another (time steps, columns,
optimisation steps), so the system of an operator is kept between prepare() calls and the
vectors come from the seed.
"""
import functools
import math

import numpy as np
import torch

import prispack_b200 as P
from prispack_b200.autograd import DiffusionPattern, SolveSpec, gaussian_random_field
from prispack_b200.autograd import solve as diff_solve

AMSED = dict(levels=3, lanczos_steps=64, low_rank=32, eig_bound=0.8, lowrank_type=0, lanczos_type=0, reorder=0)
GMSLR = dict(levels=4, low_rank=24)
PRECISION = {"f64": P.PRISM_FP64, "f32": P.PRISM_FP32, "f32apply": P.PRISM_FP32_APPLY}
KIND = {"ic": P.PRECOND_IC, "ildlt": P.PRECOND_ILDLT, "ilut": P.PRECOND_ILUT}
PECLET = 50.0  # velocity of the convection-diffusion problems along x (half along y, a quarter along z)


def listed():
    return [
        # one product with the operator of the smallest model problem: the call's own latency
        {"name": "spmv_64sq", "call": "spmv", "nx": 64, "ny": 64, "nz": 1},
        # the product with the headline operator: memory bandwidth
        {"name": "spmv_128cube", "call": "spmv", "nx": 128, "ny": 128, "nz": 128},
        # M^-1 alone, as a caller with a Krylov loop of its own uses it: threshold IC of a large 2D grid
        {"name": "apply_ic_512sq_f64", "call": "apply", "op": "poisson", "nx": 512, "ny": 512, "nz": 1,
         "precond": "ic", "precision": "f64"},
        # M^-1 of a nonsymmetric operator on a ragged 3D grid, float factor values
        {"name": "apply_ilut_61x53x47_f32", "call": "apply", "op": "convdiff", "nx": 61, "ny": 53, "nz": 47,
         "precond": "ilut", "precision": "f32"},
        # the reference's own small case: 2D Poisson 64^2, FCG + threshold IC
        {"name": "fcg_ic_64sq_f64", "call": "solve", "nx": 64, "ny": 64, "nz": 1, "precond": "ic",
         "precision": "f64"},
        # an ordinary 3D solve with the multilevel preconditioner and double factor values
        {"name": "fcg_amsed_64cube_f64", "call": "solve", "nx": 64, "ny": 64, "nz": 64, "precond": "amsed",
         "precision": "f64"},
        # the headline: 3D Poisson 128^3, multilevel preconditioner, single-precision apply
        {"name": "fcg_amsed_128cube_f32apply", "call": "solve", "nx": 128, "ny": 128, "nz": 128,
         "precond": "amsed", "precision": "f32apply"},
        # restarted FGMRES on the nonsymmetric problem
        {"name": "fgmres_gmslr_50x50x50_f32apply", "call": "fgmres", "nx": 50, "ny": 50, "nz": 50,
         "precision": "f32apply"},
        # a full block of right-hand sides that share operator and preconditioner
        {"name": "block64_ic_192sq_f32", "call": "batched", "nx": 192, "ny": 192, "k": 64, "precond": "ic",
         "precision": "f32"},
        # a narrow, odd block with the multilevel preconditioner
        {"name": "block13_amsed_95x71_f64", "call": "batched", "nx": 95, "ny": 71, "k": 13,
         "precond": "amsed", "precision": "f64"},
        # many independent systems of uneven size in one call
        {"name": "segments_48_of_32_160_f32", "call": "segments", "systems": 48, "low": 32, "high": 160,
         "precision": "f32"},
        # one step of a coefficient inversion: new coefficients, factor recomputed on the device, forward and adjoint
        {"name": "inversion_40cube_f64", "call": "inversion", "nx": 40, "ny": 40, "nz": 40},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid3(rng, lo, hi):
    s = _log_int(rng, lo, hi)
    return {a: max(4, int(s * rng.uniform(0.8, 1.0))) for a in ("nx", "ny", "nz")}


def _grid2(rng, lo, hi):
    s = _log_int(rng, lo, hi)
    return {"nx": max(8, int(s * rng.uniform(0.7, 1.0))), "ny": max(8, int(s * rng.uniform(0.7, 1.0))), "nz": 1}


def draw(rng):
    call = rng.choice(["spmv", "apply", "solve_ic", "solve_amsed", "fgmres", "batched", "segments", "inversion"])
    if call == "spmv":
        return {"call": "spmv", **(_grid3(rng, 16, 128) if rng.random() < 0.5 else _grid2(rng, 64, 1024))}
    if call == "apply":
        pc = rng.choice(["ic", "ildlt", "ilut"])
        op = "convdiff" if pc == "ilut" else "poisson"
        g = _grid3(rng, 12, 64) if op == "convdiff" or rng.random() < 0.5 else _grid2(rng, 48, 512)
        return {"call": "apply", "op": op, **g, "precond": pc, "precision": rng.choice(["f64", "f32"])}
    if call == "solve_ic":
        g = _grid3(rng, 12, 64) if rng.random() < 0.5 else _grid2(rng, 48, 400)
        return {"call": "solve", **g, "precond": "ic", "precision": rng.choice(["f64", "f32", "f32apply"])}
    if call == "solve_amsed":
        return {"call": "solve", **_grid3(rng, 24, 96), "precond": "amsed",
                "precision": rng.choice(["f64", "f32", "f32apply"])}
    if call == "fgmres":
        return {"call": "fgmres", **_grid3(rng, 20, 64), "precision": rng.choice(["f64", "f32apply"])}
    if call == "batched":
        pc = rng.choice(["ic", "amsed"])
        g = _grid2(rng, 48, 192 if pc == "ic" else 96)
        return {"call": "batched", "nx": g["nx"], "ny": g["ny"], "k": rng.randint(2, 64), "precond": pc,
                "precision": rng.choice(["f64", "f32"]) if pc == "ic" else "f64"}
    if call == "segments":
        return {"call": "segments", "systems": rng.randint(6, 48), "low": rng.randint(16, 32),
                "high": rng.randint(64, 160), "precision": rng.choice(["f64", "f32"])}
    return {"call": "inversion", **_grid3(rng, 12, 44)}


# ------------------------------------------------------------------ what a program keeps
def _key(case):
    return tuple(sorted((k, v) for k, v in case.items() if k != "name"))


def _sides(case):
    rng = np.random.default_rng(1000 * case["systems"] + case["high"])
    return [int(s) for s in rng.integers(case["low"], case["high"] + 1, size=case["systems"])]


def _base_log_kappa(case):
    return gaussian_random_field((case["nx"], case["ny"], case["nz"]), 1.0, 8.0, seed=case["nx"])


@functools.lru_cache(maxsize=16)
def _kept(key):
    """The DeviceSystem of a case's operator with its preconditioner, and what goes with it."""
    case = dict(key)
    call = case["call"]
    more = None
    if call == "segments":
        A, more = P.CSRMatrix.block_diagonal([P.CSRMatrix.laplacian(s, s, 1) for s in _sides(case)])
    elif call == "inversion":
        more = DiffusionPattern(case["nx"], case["ny"], case["nz"])
        A = more.matrix(np.exp(_base_log_kappa(case)))
    elif call == "fgmres" or case.get("op") == "convdiff":
        A = P.CSRMatrix.convection_diffusion(case["nx"], case["ny"], case["nz"], PECLET, 0.5 * PECLET, 0.25 * PECLET)
    else:
        A = P.CSRMatrix.laplacian(case["nx"], case["ny"], case.get("nz", 1))
    S = P.DeviceSystem(A, device=0)
    S.set_stream(torch.cuda.current_stream().cuda_stream)
    prec = PRECISION[case.get("precision", "f64")]
    pc = case.get("precond", "ic")
    if call == "fgmres":
        S.attach(P.HostGmslr(A, precision=prec, **GMSLR))
    elif pc == "amsed":
        S.attach(P.HostAmsed(A, precision=prec, **AMSED))
    elif call != "spmv":
        S.set_precond(KIND[pc], tol=1e-2 if pc == "ilut" else 1e-3, lfill=20, precision=prec)
    return S, more


def _vectors(case, seed, n):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    shape = (case["k"], n) if case["call"] == "batched" else (n,)
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float64)


def _target(case, seed, n):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + 7919)
    return torch.randn(n, generator=g, device="cuda", dtype=torch.float64)


def _kappa(case, seed):
    """The coefficients of one optimisation step: near those the factor's pattern was made for."""
    step = gaussian_random_field((case["nx"], case["ny"], case["nz"]), 0.1, 8.0, seed=seed % (1 << 31))
    return torch.tensor(np.exp(_base_log_kappa(case) + step), device="cuda")


def prepare(case, seed):
    S, more = _kept(_key(case))
    state = {"case": case, "S": S, "more": more, "b": _vectors(case, seed, S.n)}
    if case["call"] == "spmv":
        state["y"] = torch.empty_like(state["b"])
    if case["call"] == "inversion":
        state["kappa"] = _kappa(case, seed)
        state["target"] = _target(case, seed, S.n)
        state["spec"] = SolveSpec(tol=1e-12, max_iter=5000, refactor="device")
    return state


def run(state):
    case, S, b = state["case"], state["S"], state["b"]
    call = case["call"]
    if call == "spmv":
        return S.spmv_into(b, state["y"])
    if call == "apply":
        return S.apply(b)
    if call == "solve":
        return S.solve(b, tol=1e-10, max_iter=2000)[0]
    if call == "fgmres":
        return S.solve(b, solver=P.SOLVER_FGMRES, tol=1e-10, max_iter=1000, restart=50)[0]
    if call == "batched":
        return S.solve_batched(b, tol=1e-10, max_iter=2000)[0]
    if call == "segments":
        return S.solve_segments(state["more"], b, tol=1e-10, max_iter=2000)[0]
    kappa = state["kappa"].clone().requires_grad_(True)
    rhs = b.clone().requires_grad_(True)
    x = diff_solve(S, state["more"].values(kappa), rhs, state["spec"])
    ((x - state["target"]) ** 2).sum().backward()
    return {"x": x.detach(), "dkappa": kappa.grad, "db": rhs.grad}


# ------------------------------------------------------------------ what a pass cannot do without
def _stencil_entries(nx, ny, nz):
    return 7 * nx * ny * nz - 2 * (ny * nz + nx * nz + nx * ny) if nz > 1 else 5 * nx * ny - 2 * (nx + ny)


def work(case):
    call = case["call"]
    sizes = [(s, s, 1) for s in _sides(case)] if call == "segments" else [(case["nx"], case["ny"], case.get("nz", 1))]
    n = sum(a * b * c for a, b, c in sizes)
    nnz = sum(_stencil_entries(*s) for s in sizes)
    k = case.get("k", 1)
    vb = 8 if case.get("precision", "f64") == "f64" else 4
    matrix = 12.0 * nnz + 4.0 * n          # CSR: 8-byte values, 4-byte columns, row offsets
    factor = (4.0 + vb) * nnz + 12.0 * n   # at least the operator's own pattern
    vectors = 16.0 * n * k                 # one vector in, one out
    if call == "spmv":
        return {"bytes": matrix + vectors, "flops": 2.0 * nnz}
    if call == "apply":
        return {"bytes": factor + vectors, "flops": 2.0 * nnz}
    if call == "inversion":
        return {"bytes": 8.0 * nnz + matrix + factor + 48.0 * n, "flops": 8.0 * nnz}
    return {"bytes": matrix + factor + vectors, "flops": 4.0 * nnz * k}


# ------------------------------------------------------------------ 64-bit values
def _axis(m, axis):
    shape = [1, 1, 1]
    shape[2 - axis] = m
    return shape


def _poisson_solve(b, dims):
    """Exact inverse of the 5- / 7-point Laplacian on a Dirichlet grid by its sine eigenvectors;
    b: (..., n), x fastest."""
    d = [m for m in dims if m > 1]
    u = b.reshape((-1,) + tuple(reversed(d)))
    Q, lam = [], torch.zeros([1] * len(d), dtype=torch.float64, device=b.device)
    for a, m in enumerate(d):
        j = torch.arange(1, m + 1, dtype=torch.float64, device=b.device)
        Q.append(torch.sin(j[:, None] * j[None, :] * (math.pi / (m + 1))) * math.sqrt(2.0 / (m + 1)))
        shape = [1] * len(d)
        shape[len(d) - 1 - a] = m
        lam = lam + (4.0 * torch.sin(j * (math.pi / (2.0 * (m + 1)))) ** 2).reshape(shape)

    def modes(v):
        for a in range(len(d)):
            ax = len(d) - a  # position of axis a in v (0 is the batch)
            v = torch.movedim(torch.movedim(v, ax, -1) @ Q[a], -1, ax)
        return v
    return modes(modes(u) / lam).reshape(b.shape)


def _convdiff_product(u, dims):
    """Upwind convection-diffusion times u (nz, ny, nx)."""
    vel = (PECLET, 0.5 * PECLET, 0.25 * PECLET)
    y = torch.zeros_like(u)
    for a, m in enumerate(dims):
        c = vel[a] / (m + 1)
        ax = 2 - a
        y += (2.0 + c) * u
        y.narrow(ax, 1, m - 1).sub_(u.narrow(ax, 0, m - 1), alpha=1.0 + c)
        y.narrow(ax, 0, m - 1).sub_(u.narrow(ax, 1, m - 1))
    return y


def _poisson_product(u, dims):
    y = torch.zeros_like(u)
    for a, m in enumerate(dims):
        if m == 1:
            continue
        ax = 2 - a
        y += 2.0 * u
        y.narrow(ax, 1, m - 1).sub_(u.narrow(ax, 0, m - 1))
        y.narrow(ax, 0, m - 1).sub_(u.narrow(ax, 1, m - 1))
    return y


def _gmres(product, precond, b, restart=60, cycles=8, tol=3e-15):
    x = torch.zeros_like(b)
    nb = float(b.norm())
    best, bestx = math.inf, x
    for _ in range(cycles):
        r = b - product(x)
        beta = float(r.norm())
        if beta < best:
            best, bestx = beta, x.clone()
        else:
            break
        if beta <= tol * nb:
            break
        V, Z = [r / beta], []
        H = np.zeros((restart + 1, restart))
        for j in range(restart):
            Z.append(precond(V[j]))
            w = product(Z[j])
            for _ in range(2):
                for i in range(j + 1):
                    h = float((w * V[i]).sum())
                    H[i, j] += h
                    w = w - h * V[i]
            H[j + 1, j] = float(w.norm())
            V.append(w / H[j + 1, j])
            e = np.zeros(j + 2)
            e[0] = beta
            y, res = np.linalg.lstsq(H[:j + 2, :j + 1], e, rcond=None)[:2]
            if res.size and math.sqrt(float(res[0])) <= 1e-10 * beta:
                break
        x = x + sum(float(c) * z for c, z in zip(y, Z))
    return bestx


def _diffusion_terms(kappa, dims):
    """Face coefficients of each axis and the boundary-face term of the diagonal (kappa: nz, ny, nx)."""
    faces, bnd = [], torch.zeros_like(kappa)
    for a, m in enumerate(dims):
        ax = 2 - a
        ka, kb = kappa.narrow(ax, 0, m - 1), kappa.narrow(ax, 1, m - 1)
        faces.append(2.0 * ka * kb / (ka + kb))
        count = torch.zeros(m, dtype=kappa.dtype, device=kappa.device)
        count[0] += 1.0
        count[-1] += 1.0
        bnd = bnd + kappa * count.reshape(_axis(m, a))
    return faces, bnd


def _diffusion_form(u, v, faces, bnd, dims):
    """u . A v"""
    s = (bnd * u * v).sum()
    for a, m in enumerate(dims):
        ax = 2 - a
        s = s + (faces[a] * (u.narrow(ax, 1, m - 1) - u.narrow(ax, 0, m - 1))
                 * (v.narrow(ax, 1, m - 1) - v.narrow(ax, 0, m - 1))).sum()
    return s


def _diffusion_solve(b, faces, bnd, dims):
    """Conjugate gradients with the diagonal, refined to the rounding of 64 bits."""
    diag = bnd.clone()
    for a, m in enumerate(dims):
        diag.narrow(2 - a, 0, m - 1).add_(faces[a])
        diag.narrow(2 - a, 1, m - 1).add_(faces[a])

    def product(u):
        y = bnd * u
        for a, m in enumerate(dims):
            ax = 2 - a
            f = faces[a] * (u.narrow(ax, 1, m - 1) - u.narrow(ax, 0, m - 1))
            y.narrow(ax, 1, m - 1).add_(f)
            y.narrow(ax, 0, m - 1).sub_(f)
        return y
    x = torch.zeros_like(b)
    for _ in range(3):
        r = b - product(x)
        z = r / diag
        p, rz, stop = z.clone(), (r * z).sum(), 1e-11 * float(r.norm())
        for it in range(4000):
            q = product(p)
            alpha = rz / (p * q).sum()
            x = x + alpha * p
            r = r - alpha * q
            if it % 20 == 19 and float(r.norm()) <= stop:
                break
            z = r / diag
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
    return x


def exact(case, seed):
    call = case["call"]
    if call == "apply":
        return None  # what M is depends on the threshold factorisation itself
    if call == "segments":
        n = sum(s * s for s in _sides(case))
        b, parts, at = _vectors(case, seed, n), [], 0
        for s in _sides(case):
            parts.append(_poisson_solve(b[at:at + s * s], (s, s, 1)))
            at += s * s
        return torch.cat(parts)
    dims = (case["nx"], case["ny"], case.get("nz", 1))
    n = dims[0] * dims[1] * dims[2]
    b = _vectors(case, seed, n)
    grid = (dims[2], dims[1], dims[0])
    if call == "spmv":
        return _poisson_product(b.reshape(grid), dims).reshape(-1)
    if call == "fgmres":
        return _gmres(lambda u: _convdiff_product(u, dims), lambda u: _poisson_solve(u.reshape(-1), dims).reshape(grid),
                      b.reshape(grid)).reshape(-1)
    if call == "inversion":
        kappa = _kappa(case, seed).reshape(grid)
        faces, bnd = _diffusion_terms(kappa, dims)
        x = _diffusion_solve(b.reshape(grid), faces, bnd, dims)
        lam = _diffusion_solve(2.0 * (x - _target(case, seed, n).reshape(grid)), faces, bnd, dims)
        k = kappa.clone().requires_grad_(True)
        f, d = _diffusion_terms(k, dims)
        (-_diffusion_form(lam, x, f, d, dims)).backward()
        return {"x": x.reshape(-1), "dkappa": k.grad.reshape(-1), "db": lam.reshape(-1)}
    return _poisson_solve(b, dims)
