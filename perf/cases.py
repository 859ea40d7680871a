"""Timed cases of the solver: what the programs that use it have it do, over the sizes they do it at.

Six kinds of pass, each through the public entry points:

* ``newton`` — new values on a known pattern, then a solve, both in device memory
  (``Handle.refactor_device`` + ``solve_device``): one Newton iteration or load step;
* ``step``   — a solve with a factor that is kept (``solve_device``): one time step of a linear
  dynamic or thermal analysis;
* ``batch``  — the same as ``newton`` for many independent plates in one forest (``factor_batch``);
* ``engine`` — the engine's solver API: K assembled on the device from C3D8 elements, factored and
  solved for a host load vector (``SystemMatrix`` / ``Assembly``);
* ``call``   — the C interface as a plug-in calls it, all host buffers: ``rustyfem_factor``,
  ``rustyfem_solve``, ``rustyfem_free``;
* ``indef`` and ``unsym`` — the same call for symmetric indefinite systems (a Laplacian shifted into
  its spectrum, as an eigenvalue solver or a Sturm check factors it) and for unsymmetric ones
  (a tangent with friction or follower loads).

The right-hand sides belong to known solutions: a smooth displacement field (a polynomial that
vanishes at the clamped face, with one percent of noise) times the matrix. The smooth part is what
loads excite, and it is the part that the conditioning of the matrix makes hard.
"""
from __future__ import annotations

import dataclasses
import functools
import math

import numpy as np
import torch

from rustyfem_b200 import ffi, solver, workloads

PRECISION = {"fp64": ffi.FP64, "mixed": ffi.MIXED}


def listed():
    return [
        # the smallest call: a time step of a 2D strip of a few hundred equations; latency only
        dict(name="step_plate_41x4", kind="step", mesh="plate", nx=41, ny=4, precision="fp64", nrhs=1),
        # time stepping of a solid of 114,444 equations with the FP64 factor
        dict(name="step_hex8_33_fp64", kind="step", mesh="hex8", nx=33, precision="fp64", nrhs=1),
        # Newton iterations of a small, an ordinary and two large solids; 60³ in mixed precision is
        # the model of the benchmark, 45³ in FP64 the largest that most FP64 users run
        dict(name="newton_hex8_9_fp64", kind="newton", mesh="hex8", nx=9, precision="fp64", nrhs=1),
        dict(name="newton_hex8_22_fp64", kind="newton", mesh="hex8", nx=22, precision="fp64", nrhs=1),
        dict(name="newton_hex8_45_fp64", kind="newton", mesh="hex8", nx=45, precision="fp64", nrhs=1),
        dict(name="newton_hex8_60_mixed", kind="newton", mesh="hex8", nx=60, precision="mixed", nrhs=1),
        # quadratic elements with many load cases at once
        dict(name="newton_hex20_20_mixed_32rhs", kind="newton", mesh="hex20", nx=20, precision="mixed", nrhs=32),
        # parameter study: many small 2D models with a few load cases each, one forest
        dict(name="batch_plates_160_fp64_8rhs", kind="batch", models=160, lo=20, hi=200, precision="fp64", nrhs=8),
        # the engine's loop: assembly, factor, solve (leaf size 48)
        dict(name="engine_hex8_30_fp64", kind="engine", mesh="hex8", nx=30),
        # a plug-in's whole call on host buffers, analysis included
        dict(name="call_hex8_20_fp64", kind="call", mesh="hex8", nx=20),
        # eigenvalue solver: shifted Laplacian, about a tenth of the spectrum below the shift
        dict(name="indef_laplace_24", kind="indef", nx=24),
        # unsymmetric tangent with delayed pivots
        dict(name="unsym_hex8_13", kind="unsym", mesh="hex8", nx=13, alpha=10.0),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["step", "newton", "newton", "batch", "engine", "call", "indef", "unsym"])
    if kind == "batch":
        lo = rng.randint(4, 60)
        return dict(kind=kind, models=_log_int(rng, 6, 160), lo=lo, hi=rng.randint(lo + 20, 200),
                    precision="fp64", nrhs=rng.choice([1, 2, 3, 5, 8]))
    if kind == "engine":
        return dict(kind=kind, mesh="hex8", nx=_log_int(rng, 4, 38))
    if kind == "call":
        return dict(kind=kind, mesh="hex8", nx=_log_int(rng, 4, 24))
    if kind == "indef":
        return dict(kind=kind, nx=rng.randint(6, 24))
    if kind == "unsym":
        return dict(kind=kind, mesh="hex8", nx=rng.randint(4, 13), alpha=rng.choice([0.5, 10.0, 30.0]))
    mesh = rng.choice(["hex8", "hex8", "hex20", "plate"])
    case = dict(kind=kind, mesh=mesh, precision=rng.choice(["fp64", "mixed"]),
                nrhs=rng.choice([1, 1, 1, 2, 4, 7, 8, 13, 32]))
    if mesh == "hex8":
        case["nx"] = _log_int(rng, 4, 45)
    elif mesh == "hex20":
        case["nx"] = _log_int(rng, 3, 20)
    else:
        case["nx"] = _log_int(rng, 20, 200)
        case["ny"] = max(2, case["nx"] // 10)
        case["precision"] = "fp64"   # what RFG_AUTO takes for small fronts
    return case


# --- meshes and matrices ---------------------------------------------------------------------

CORNER = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1],
                   [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], float)


@functools.lru_cache(maxsize=None)
def _ke_hex8(h, nu):
    """Stiffness of a cubic element of edge h for E = 1 (2×2×2 points, mean dilatation)."""
    lam, mu = nu / ((1 + nu) * (1 - 2 * nu)), 0.5 / (1 + nu)
    D = np.zeros((6, 6))
    D[:3, :3] = lam
    D[np.arange(6), np.arange(6)] += [2 * mu] * 3 + [mu] * 3
    B = []
    for q in CORNER / math.sqrt(3.0):
        dn = np.empty((8, 3))
        for a in range(3):
            o = [c for c in range(3) if c != a]
            dn[:, a] = CORNER[:, a] * np.prod(1 + q[o] * CORNER[:, o], axis=1) / 8 * (2 / h)
        b = np.zeros((6, 24))
        for a in range(3):
            b[a, a::3] = dn[:, a]
        for r, (i, j) in enumerate([(0, 1), (1, 2), (0, 2)]):
            b[3 + r, i::3] = dn[:, j]
            b[3 + r, j::3] = dn[:, i]
        B.append(b)
    vol = [b[:3].sum(0) for b in B]
    mean = sum(vol) / 8
    K = np.zeros((24, 24))
    for b, v in zip(B, vol):
        b = b.copy()
        b[:3] += (mean - v) / 3
        K += b.T @ D @ b * (h / 2) ** 3
    return K


def _hex8_graph(n):
    """Node graph of the free nodes (x > 0) of an n³ cube, nodes numbered x fastest."""
    p = n + 1
    k, j, i = (a.ravel() for a in np.meshgrid(np.arange(p), np.arange(p), np.arange(1, p), indexing="ij"))
    nbr = np.full((len(i), 27), -1, np.int64)
    for s in range(27):
        a, b, c = i + s % 3 - 1, j + s // 3 % 3 - 1, k + s // 9 - 1
        ok = (a >= 1) & (a <= n) & (b >= 0) & (b <= n) & (c >= 0) & (c <= n) & (s != 13)
        nbr[ok, s] = ((c * p + b) * n + a - 1)[ok]
    ptr = np.concatenate([[0], np.cumsum((nbr >= 0).sum(1))]).astype(np.int64)
    return workloads.Graph(np.stack([i, j, k], 1) / n, ptr, nbr[nbr >= 0], np.full(len(i), 3, np.int64))


@functools.lru_cache(maxsize=1)
def _hex8_mesh(n):
    return workloads.hex8_mesh(n)


def _moduli(n, seed):
    """Young's modulus per element: steel that has softened by up to a half in places."""
    return 210e9 * np.random.default_rng([seed, 1]).uniform(0.5, 1.0, n ** 3)


def _hex8_edof(n):
    mesh = _hex8_mesh(n)
    return mesh.edof(3 * np.arange(n * (n + 1) ** 2))


def _hex8_model(n, emod):
    """The cube as a caller of the C interface has it: both triangles in CSC, free DOFs only."""
    edof = torch.from_numpy(_hex8_edof(n)).cuda()
    N = 3 * n * (n + 1) ** 2
    rows = edof[:, :, None].expand(-1, 24, 24).reshape(-1)
    cols = edof[:, None, :].expand(-1, 24, 24).reshape(-1)
    ke = torch.from_numpy(_ke_hex8(1.0 / n, 0.3)).cuda()
    vals = (torch.from_numpy(emod).cuda()[:, None, None] * ke).reshape(-1)
    ok = (rows >= 0) & (cols >= 0)
    A = torch.sparse_coo_tensor(torch.stack([rows[ok], cols[ok]]), vals[ok], (N, N)).coalesce().to_sparse_csr()
    mesh = _hex8_mesh(n)
    free = np.flatnonzero(mesh.block >= 0)
    return workloads.Model(f"hex8 {n}^3", N, len(mesh.xyz), np.repeat(free, 3), mesh.xyz.ravel(),
                           A.crow_indices().cpu().numpy(), A.col_indices().cpu().numpy(), A.values().cpu().numpy(),
                           np.zeros(N), symmetric_storage="full")


def _hex8_load(n, emod, u):
    """K·u for one displacement vector (caller's numbering), element by element."""
    edof = _hex8_edof(n)
    ue = np.where(edof >= 0, u[np.maximum(edof, 0)], 0.0)
    fe = (ue @ _ke_hex8(1.0 / n, 0.3)) * emod[:, None]
    ok = edof >= 0
    return np.bincount(edof[ok], weights=fe[ok], minlength=len(u))


@functools.lru_cache(maxsize=8)
def _hex20(n):
    return workloads.hex20_cube(n).full()


@functools.lru_cache(maxsize=512)
def _plate(nx, ny):
    return workloads.plate(nx, ny).full()


def _plate_sizes(case):
    return workloads.plate_sizes(case["models"], seed=11, lo=case["lo"], hi=case["hi"])


def _scaled(model, seed):
    """The model with another Young's modulus."""
    e = np.random.default_rng([seed, 2]).uniform(1 / 3, 1.0)
    return dataclasses.replace(model, data=model.data * e)


def _product(model, X):
    """(nrhs, n) right-hand sides A·x for the rows x of X. A is given by columns, so its transpose
    by rows; ``model`` holds both triangles."""
    A = torch.sparse_csr_tensor(torch.from_numpy(model.indptr), torch.from_numpy(model.indices),
                                torch.from_numpy(model.data), (model.n, model.n)).cuda()
    if model.name.endswith("unsym"):
        A = A.to_sparse_coo().t().coalesce().to_sparse_csr()
    return (A @ torch.from_numpy(np.ascontiguousarray(X.T)).cuda()).T.contiguous()


def _field(loc, xyz, nrhs, seed):
    """(nrhs, n) displacement vectors: a quadratic field that vanishes at x = 0, and noise."""
    rng = np.random.default_rng([seed, 3])
    x, y, z = xyz.reshape(-1, 3)[loc].T / xyz.max()
    base = x * np.stack([np.ones_like(x), x, y, z, x * x, x * y, y * z, z * x])
    comp = np.arange(len(loc)) - np.searchsorted(loc, loc)
    out = np.empty((nrhs, len(loc)))
    for r in range(nrhs):
        c = rng.uniform(-1e-3, 1e-3, (3, len(base)))
        for a in range(3):
            m = comp == a
            out[r, m] = c[a] @ base[:, m]
    return out + 1e-5 * rng.standard_normal(out.shape)


def _model(case, seed):
    if case["kind"] == "indef":
        m, _ = workloads.laplace3d(case["nx"], workloads.laplace_sigma(case["nx"]))
        m = m.full()
        e = np.random.default_rng([seed, 2]).uniform(0.5, 2.0)
        return dataclasses.replace(m, data=m.data * e)
    if case["kind"] == "unsym":
        m = workloads.skew_perturbed(_hex8_model(case["nx"], _moduli(case["nx"], seed)), case["alpha"], seed)
        return dataclasses.replace(m, name=m.name + " unsym")
    if case["mesh"] == "hex8":
        return _hex8_model(case["nx"], _moduli(case["nx"], seed))
    if case["mesh"] == "hex20":
        return _scaled(_hex20(case["nx"]), seed)
    return _scaled(_plate(case["nx"], case["ny"]), seed)


def _solution(case, seed):
    """(nrhs, n) known solutions in the caller's numbering."""
    nrhs = case.get("nrhs", 1)
    if case["kind"] == "batch":
        parts = []
        for i, (nx, ny) in enumerate(_plate_sizes(case)):
            p = _plate(nx, ny)
            parts.append(_field(p.loc, p.coords, nrhs, 1000 * seed + i))
        return np.concatenate(parts, axis=1)
    if case["kind"] == "indef":
        return np.random.default_rng([seed, 4]).standard_normal((1, case["nx"] ** 3))
    if case["mesh"] == "hex8":
        mesh = _hex8_mesh(case["nx"])
        return _field(np.repeat(np.flatnonzero(mesh.block >= 0), 3), mesh.xyz.ravel(), nrhs, seed)
    p = _hex20(case["nx"]) if case["mesh"] == "hex20" else _plate(case["nx"], case["ny"])
    return _field(p.loc, p.coords, nrhs, seed)


# --- the passes ------------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "engine":
        n = case["nx"]
        mesh, emod = _hex8_mesh(n), _moduli(n, seed)
        matrix = solver.select("direct-gpu").prepare(_hex8_graph(n))
        asm = matrix.assembly(mesh.edof(matrix.first_dof()))
        f = _hex8_load(n, emod, _solution(case, seed)[0])
        b = np.empty_like(f)
        b[(matrix.first_dof()[:, None] + np.arange(3)).ravel()] = f
        return dict(case=case, matrix=matrix, asm=asm, mesh=mesh, emod=emod, b=b)
    X = _solution(case, seed)
    if kind == "batch":
        models = [_scaled(_plate(nx, ny), 1000 * seed + i) for i, (nx, ny) in enumerate(_plate_sizes(case))]
        off = np.concatenate([[0], np.cumsum([m.n for m in models])])
        b = torch.cat([_product(m, X[:, off[i]:off[i + 1]]) for i, m in enumerate(models)], dim=1).contiguous()
        h, _, _ = ffi.factor_batch(models, precision=PRECISION[case["precision"]])
        values = torch.from_numpy(np.concatenate([m.data for m in models])).cuda()
        return dict(case=case, handle=h, values=values, b=b, x=torch.empty_like(b))
    model = _model(case, seed)
    if case.get("mesh") == "hex8" and kind != "unsym":
        emod = _moduli(case["nx"], seed)
        b = torch.from_numpy(np.stack([_hex8_load(case["nx"], emod, u) for u in X])).cuda()
    else:
        b = _product(model, X)
    if kind in ("call", "indef", "unsym"):
        return dict(case=case, model=model, b=b.cpu().numpy()[0].copy())
    h, err, _ = ffi.factor(model, precision=PRECISION[case["precision"]])
    assert h is not None, f"not positive definite at DOF {err}"
    return dict(case=case, handle=h, values=torch.from_numpy(model.data).cuda(), b=b, x=torch.empty_like(b))


def run(state):
    kind = state["case"]["kind"]
    if kind == "engine":
        m, mesh = state["matrix"], state["mesh"]
        state["asm"].hex8(mesh.xyz, mesh.conn, state["emod"], mesh.nu)
        m.factor()
        x = state["b"].copy()
        m.solve(x)
        return x
    if kind == "call":
        h, _, d = ffi.factor(state["model"], want_d=True)
        x = h.solve(state["b"])
        h.free()
        return x, d
    if kind == "indef":
        h, _, inertia = ffi.factor_indef(state["model"])
        x = h.solve(state["b"])
        h.free()
        return x, np.array(inertia)
    if kind == "unsym":
        h, _, _ = ffi.factor_unsym(state["model"])
        x = h.solve(state["b"])
        h.free()
        return x
    h, x = state["handle"], state["x"]
    if kind in ("newton", "batch"):
        h.refactor_device(state["values"].data_ptr())
    x.copy_(state["b"])
    h.solve_device(x.data_ptr(), x.shape[0])
    return x


def exact(case, seed):
    if case["kind"] == "engine":
        return None   # the solver numbers the equations
    X = _solution(case, seed)
    if case["kind"] == "call":
        return X[0], None
    if case["kind"] == "indef":
        return X[0], None
    return X[0] if case["kind"] == "unsym" else X


# --- the work of a pass ----------------------------------------------------------------------

def _laplace_graph(g):
    v = np.arange(g ** 3)
    i, j, k = v % g, v // g % g, v // (g * g)
    nbr = np.full((len(v), 6), -1, np.int64)
    for s, (a, off) in enumerate([(k, -g * g), (j, -g), (i, -1), (i, 1), (j, g), (k, g * g)]):
        ok = (a > 0) if off < 0 else (a < g - 1)
        nbr[ok, s] = v[ok] + off
    ptr = np.concatenate([[0], np.cumsum((nbr >= 0).sum(1))]).astype(np.int64)
    return workloads.Graph(np.stack([i, j, k], 1).astype(float), ptr, nbr[nbr >= 0], np.ones(len(v), np.int64))


@functools.lru_cache(maxsize=64)
def _size(mesh, nx, ny, leaf):
    """(equations, entries of the lower triangle, flops and entries of the factor)."""
    if mesh == "hex8":
        g = _hex8_graph(nx)
    elif mesh == "laplace":
        g = _laplace_graph(nx)
    else:
        g = (_hex20(nx) if mesh == "hex20" else _plate(nx, ny)).graph
    S = ffi.Symbolic(g, leaf)
    d = int(g.ndof[0])
    n = S.n
    return n, (len(g.adj_idx) * d * d + n * d + n) // 2, S.work(), S.factor_size()


def work(case):
    """The values, the right-hand sides and the solutions once; a kept factor is an input of the
    solve. Two triangles (LU) cost and hold twice as much."""
    kind, nrhs = case["kind"], case.get("nrhs", 1)
    if kind == "batch":
        sizes = [_size("plate", nx, ny, 16) for nx, ny in _plate_sizes(case)]
        n, nnz, flops, nl = (sum(s[q] for s in sizes) for q in range(4))
    else:
        n, nnz, flops, nl = _size(case.get("mesh", "laplace"), case["nx"], case.get("ny", 0),
                                  48 if kind == "engine" else 16)
    two = 2 if kind == "unsym" else 1
    vectors = 16 * n * nrhs
    solve = 4.0 * nl * nrhs * two
    if kind == "step":
        return {"bytes": nl * (4 if case["precision"] == "mixed" else 8) + vectors, "flops": solve}
    return {"bytes": 8 * nnz * two + vectors, "flops": flops * two + solve}
