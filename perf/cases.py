"""Performance cases: the solves that a program has this library do.

A case is one system (how its matrix is made, its size, the precision) and one
call pattern on it:

* ``step``    -- a Newton step's linear solve: the pattern was analysed before,
  new values arrive in device memory, ``factorize_device`` + ``solve_device``;
* ``solve``   -- a further right-hand side on a factorized system (time
  stepping with a constant matrix): ``solve_device`` alone;
* ``host``    -- the polysolve calls on host arrays: ``factorize`` + ``solve``;
* ``adjoint`` -- ``lss.autograd``: forward solve of A(theta) x = b and the
  backward pass to dL/dtheta and dL/db;
* ``batch``   -- ``lss.Batch``: several systems x 16 right-hand sides.

Systems: P1-tet elasticity on nx x ny x nz node grids (block size 3) with
lognormal moduli and penalty springs or with a stiff spherical inclusion, and
scalar Laplacians on Delaunay triangulations with collapsed triangles (block
size 1).  Tolerances are the library's default (relative residual 1e-10).
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "local-stiff-solver_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import lss  # noqa: E402
from lss import autograd, gen  # noqa: E402

RHS = 16  # right-hand sides per system of a batch


def listed():
    cube = {"system": "cube", "springs": 0.01, "contrast": 1.0}
    ball = {"system": "cube", "springs": 0.0}
    return [
        # the smallest calls, where latency and launches count: a coarse 2D
        # mesh through the host interface, a coarse cube inside a Newton loop
        {"name": "laplace_3k_fp64_host", "system": "laplace", "points": 3001, "precision": "fp64", "call": "host"},
        {"name": "cube_2k_fp64_step", **cube, "nx": 9, "ny": 9, "nz": 9, "precision": "fp64", "call": "step"},
        # ordinary sizes: a cube with a stiff inclusion in default precision, a
        # further right-hand side on one in mixed precision, a ragged box
        {"name": "ball_24k_fp64_step", **ball, "contrast": 1e6, "nx": 20, "ny": 20, "nz": 20, "precision": "fp64",
         "call": "step"},
        {"name": "ball_34k_mixed_solve", **ball, "contrast": 1e4, "nx": 23, "ny": 21, "nz": 24, "precision": "mixed",
         "call": "solve"},
        {"name": "ball_81k_mixed_step", **ball, "contrast": 1e4, "nx": 31, "ny": 30, "nz": 29, "precision": "mixed",
         "call": "step"},
        {"name": "cube_206k_mixed_host", **cube, "nx": 43, "ny": 37, "nz": 43, "precision": "mixed", "call": "host"},
        # large 3D systems, default and mixed precision
        {"name": "cube_648k_fp64_step", **cube, "nx": 60, "ny": 60, "nz": 60, "precision": "fp64", "call": "step"},
        {"name": "cube_3m_mixed_step", **cube, "nx": 100, "ny": 100, "nz": 100, "precision": "mixed", "call": "step"},
        # 2D meshes with bad triangles: many stiff subdomains, thousands of short iterations
        {"name": "laplace_60k_mixed_solve", "system": "laplace", "points": 60013, "precision": "mixed",
         "call": "solve"},
        {"name": "laplace_150k_fp64_step", "system": "laplace", "points": 150000, "precision": "fp64",
         "call": "step"},
        # differentiation: one Young's modulus per element, forward + backward
        {"name": "adjoint_24k_mixed", "system": "parametric", "nodes": 20, "contrast": 1e5, "precision": "mixed",
         "call": "adjoint"},
        # throughput: several systems of different sizes, 16 right-hand sides each
        {"name": "batch_6x16_mixed", "system": "batch", "count": 6, "dofs_lo": 5000, "dofs_hi": 60000,
         "precision": "mixed", "call": "batch"},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["laplace", "cube", "cube", "ball", "ball", "parametric", "batch"])
    precision = rng.choice(["fp64", "mixed"])
    call = rng.choice(["step", "step", "solve", "host"])
    if kind == "laplace":
        return {"system": "laplace", "points": int(_log_uniform(rng, 1000, 150000)), "precision": precision,
                "call": call}
    if kind == "parametric":
        return {"system": "parametric", "nodes": rng.randint(8, 20), "contrast": 10.0 ** rng.uniform(3, 5),
                "precision": precision, "call": "adjoint"}
    if kind == "batch":
        lo = int(_log_uniform(rng, 2000, 10000))
        return {"system": "batch", "count": rng.randint(2, 6), "dofs_lo": lo, "dofs_hi": lo * rng.randint(2, 6),
                "precision": "mixed", "call": "batch"}
    hi = 40 if kind == "ball" else (60 if precision == "fp64" else 80)
    m = _log_uniform(rng, 8, hi)  # nodes per side, each side up to a tenth longer or shorter
    nx, ny, nz = (max(6, int(m * rng.uniform(0.9, 1.1))) for _ in range(3))
    return {"system": "cube", "springs": 0.01 if kind == "cube" else 0.0,
            "contrast": 1.0 if kind == "cube" else 10.0 ** rng.uniform(3, 6), "nx": nx, "ny": ny, "nz": nz,
            "precision": precision, "call": call}


# ---------------------------------------------------------------- systems

def _matrix(case, seed):
    """(A, b, GPUHybrid parameters) of a single system."""
    rng = np.random.Generator(np.random.PCG64(seed))
    if case["system"] == "laplace":
        A, _ = gen.laplacian_delaunay(case["points"], rng)
        return A, rng.standard_normal(A.shape[0]), {"block_size": 1, "max_iter": 50000}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["springs"] > 0:
        E = rng.lognormal(0.0, 1.0, size=6 * (nx - 1) * (ny - 1) * (nz - 1))
        top = np.arange(nx * ny, dtype=np.int64) + (nz - 1) * nx * ny
        nodes = rng.choice(top, size=max(1, round(case["springs"] * len(top))), replace=False)
        A = gen.elasticity_cube(nx, ny, nz, E, spring_nodes=np.sort(nodes).astype(np.int32))
        params = {"block_size": 3, "max_iter": 20000, "decompose_subdomains": False}
    else:
        E, _ = gen.sphere_inclusion_E(nx, ny, nz, rng, E_in=case["contrast"])
        A = gen.elasticity_cube(nx, ny, nz, E)
        params = {"block_size": 3, "max_iter": 20000, "gmm_jump_threshold": 10.0, "min_subdomain_size": 4}
    return A, rng.standard_normal(A.shape[0]), params


def _ball_params():
    return {"block_size": 3, "max_iter": 20000, "gmm_jump_threshold": 10.0, "min_subdomain_size": 4}


def _parametric(case, seed):
    """(pattern, M, c, theta, b, x*): A(theta).data = M theta + c, L = |x - x*|^2 / 2."""
    nodes = case["nodes"]
    rng = np.random.Generator(np.random.PCG64(seed))
    pattern, M, c = gen.elasticity_parametric(nodes)
    E, _ = gen.sphere_inclusion_E(nodes, nodes, nodes, rng, radius=0.2, E_in=case["contrast"])
    theta = E * rng.lognormal(0.0, 1.0, size=len(E))
    n = pattern.shape[0]
    return pattern, M, c, theta, rng.standard_normal(n), rng.standard_normal(n)


def _batch_systems(case, seed):
    """[(A, B)]: cubes of sizes spread over [dofs_lo, dofs_hi], inclusions of contrasts 1e3 to 1e5."""
    rng = np.random.Generator(np.random.PCG64(seed))
    out = []
    for s in range(case["count"]):
        t = s / max(1, case["count"] - 1)
        m = max(4, round((case["dofs_lo"] * (case["dofs_hi"] / case["dofs_lo"]) ** t / 3.0) ** (1.0 / 3.0)))
        E, _ = gen.sphere_inclusion_E(m, m, m, rng, E_in=10.0 ** rng.uniform(3.0, 5.0))
        A = gen.elasticity_cube(m, m, m, E)
        out.append((A, rng.standard_normal((RHS, A.shape[0]))))
    return out


def _solver_params(params, case):
    return {"solver": "GPUHybrid", "GPUHybrid": params, "gb300": {"precision": case["precision"]}}


def _device(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# ---------------------------------------------------------------- the calls

def prepare(case, seed):
    call = case["call"]
    st = {"call": call, "stream": torch.cuda.Stream()}
    if call == "adjoint":
        pattern, M, c, theta, b, target = _parametric(case, seed)
        st["system"] = autograd.LinearSystem(pattern, M, c, _solver_params(_ball_params(), case))
        st["theta"] = _device(theta).requires_grad_(True)
        st["b"] = _device(b).requires_grad_(True)
        st["target"] = _device(target)
    elif call == "batch":
        st["solvers"], st["values"], st["b"], st["x"] = [], [], [], []
        for A, B in _batch_systems(case, seed):
            s = lss.Solver.create(_solver_params(_ball_params(), case))
            s.analyze_pattern(A)
            st["solvers"].append(s)
            st["values"].append(_device(A.data))
            st["b"].append(_device(B))
            st["x"].append(torch.zeros_like(st["b"][-1]))
        st["batch"] = lss.Batch(st["solvers"])
    else:
        A, b, params = _matrix(case, seed)
        s = lss.Solver.create(_solver_params(params, case))
        s.analyze_pattern(A)
        st["solver"] = s
        if call == "host":
            st["A"], st["b"] = A, b
        else:
            st["values"], st["b"] = _device(A.data), _device(b)
            st["x"] = torch.zeros_like(st["b"])
            if call == "solve":
                torch.cuda.synchronize()
                s.factorize_device(st["values"].data_ptr(), st["stream"].cuda_stream)
    torch.cuda.synchronize()
    return st


def run(st):
    call = st["call"]
    if call == "host":
        st["solver"].factorize(st["A"])
        return st["solver"].solve(st["b"])
    if call == "batch":
        for x in st["x"]:
            x.zero_()
        torch.cuda.current_stream().synchronize()
        st["batch"].factorize_device([v.data_ptr() for v in st["values"]])
        st["batch"].solve_device([b.data_ptr() for b in st["b"]], [x.data_ptr() for x in st["x"]])
        return list(st["x"])
    with torch.cuda.stream(st["stream"]):
        h = st["stream"].cuda_stream
        if call == "adjoint":
            theta, b = st["theta"], st["b"]
            theta.grad = b.grad = None
            x = autograd.solve(theta, b, st["system"])
            (0.5 * ((x - st["target"]) ** 2).sum()).backward()
            return {"x": x.detach(), "dtheta": theta.grad, "db": b.grad}
        st["x"].zero_()
        if call == "step":
            st["solver"].factorize_device(st["values"].data_ptr(), h)
        st["solver"].solve_device(st["b"].data_ptr(), st["x"].data_ptr(), h)
        return st["x"]


# ---------------------------------------------------------------- sizes and values

def _sizes(case):
    """(unknowns, stored entries, values in, values out) of one pass, in numbers."""
    if case["system"] == "laplace":
        n = case["points"]
        nnz = 7.0 * n
        return n, nnz, n, n
    if case["system"] == "batch":
        n = 0.0
        for s in range(case["count"]):
            t = s / max(1, case["count"] - 1)
            n += case["dofs_lo"] * (case["dofs_hi"] / case["dofs_lo"]) ** t
        return n, 36.0 * n, RHS * n, RHS * n
    if case["system"] == "parametric":
        m = case["nodes"]
        n, ne = 3.0 * m ** 3, 6.0 * (m - 1) ** 3
        return n, 36.0 * n, 2 * n + ne, 2 * n + ne
    n = 3.0 * case["nx"] * case["ny"] * case["nz"]
    return n, 36.0 * n, n, n


def work(case):
    """The matrix values, the right-hand sides and the results once, and one
    product with the matrix per right-hand side."""
    n, nnz, vin, vout = _sizes(case)
    products = {"batch": RHS, "adjoint": 2}.get(case["call"], 1)
    return {"bytes": 8.0 * (nnz + vin + vout), "flops": 2.0 * nnz * products}


def _cg(A, b):
    """A x = b in 64 bits by diagonally scaled conjugate gradients with
    restarts from the true residual, on torch's sparse product; b: (k, n), k
    right-hand sides side by side."""
    T = torch.sparse_csr_tensor(_device(A.indptr.astype(np.int64)), _device(A.indices.astype(np.int64)),
                                _device(np.asarray(A.data, np.float64)), size=A.shape)
    d = _device(np.asarray(A.diagonal(), np.float64))[:, None]
    b = _device(b.T)
    x, best, floor = torch.zeros_like(b), None, 1e-9 * torch.linalg.vector_norm(b, dim=0)
    for _ in range(6):
        r = b - T @ x
        norm = torch.linalg.vector_norm(r, dim=0)
        if best is not None and float((norm / best).max()) > 0.5:
            break
        best = norm
        stop = torch.minimum(floor, 1e-6 * norm)
        e, z = torch.zeros_like(b), r / d
        p, g = z.clone(), (r * z).sum(0)
        for k in range(30000):
            q = T @ p
            a = g / (p * q).sum(0).clamp_min(1e-300)
            e += a * p
            r -= a * q
            z = r / d
            g, old = (r * z).sum(0), g
            p = z + (g / old.clamp_min(1e-300)) * p
            if k % 50 == 49 and bool((torch.linalg.vector_norm(r, dim=0) <= stop).all()):
                break
        x = x + e
    return x.T.contiguous()


def exact(case, seed):
    if case["call"] == "batch":
        return [_cg(A, B) for A, B in _batch_systems(case, seed)]
    if case["call"] == "adjoint":
        pattern, M, c, theta, b, target = _parametric(case, seed)
        A = pattern.copy()
        A.data = M @ theta + c
        x = _cg(A, b[None])[0].cpu().numpy()
        lam = _cg(A, (x - target)[None])[0].cpu().numpy()
        rows = np.repeat(np.arange(A.shape[0]), np.diff(A.indptr))
        return {"x": x, "dtheta": M.T @ (-lam[rows] * x[A.indices]), "db": lam}
    A, b, _ = _matrix(case, seed)
    x = _cg(A, b[None])[0]
    return x.cpu().numpy() if case["call"] == "host" else x
