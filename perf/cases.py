"""The solves that programs ask of this package, as cases to time.

A case is one linear system (or a set of them) with its controls: 2-D P1
Poisson and 3-D log-normal diffusion from the smallest grids of the tests to
the benchmark's 128^3, several right-hand sides at once, batches of uneven
independent systems, elemental elasticity with the rigid-body coarse space,
a training step through the differentiable solve and the plain CSR residual.
``prepare`` leaves a program where it stands before the call: matrix set,
``setup`` done, right-hand side in hand.  ``run`` is the call: the numeric
factorisations and the PCG iterations (with ``reuse`` the iterations alone:
the factors of an earlier solve are kept), or for ``adjoint`` the whole
forward and backward pass with its own setup.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from doug_gb300 import DougSolver, residual_csr
from doug_gb300 import problems as P

BASE = dict(solver=2, method=1, fine_method=1, levels=2, smoothers=1, strong1="0.08")
# 3-D diffusion: the benchmark's controls; 2-D, batches and elasticity: the
# controls of the small, batched and elemental benchmark lines
CTL3 = dict(BASE, overlap=2, radius1=5, maxasize1=400, solve_tolerance="1.0e-8", solve_maxiters=2000)
CTL2 = dict(BASE, overlap=1, radius1=2, solve_tolerance="1.0e-8", solve_maxiters=3000)
CTLE = dict(BASE, overlap=1, radius1=2, maxasize1=100, coarse_method=3, solve_tolerance="1.0e-8", solve_maxiters=5000)
CTLA = dict(CTL2, solve_tolerance="1.0e-10")


def listed():
    return [
        # a user's first and smallest system, host buffers in and out, FP64 as by default: launches and latency
        {"name": "poisson2d_33_host", "kind": "poisson2d", "nodes": 33, "parts": 0, "mixed": False, "nrhs": 1, "reuse": False, "host": True},
        # the small plain benchmark case: 16,129 unknowns, four imported quadrants, FP64
        {"name": "poisson2d_129", "kind": "poisson2d", "nodes": 129, "parts": 2, "mixed": False, "nrhs": 1, "reuse": False, "host": False},
        # an ordinary 2-D system of odd size in mixed precision, nine ragged parts
        {"name": "poisson2d_271_mixed", "kind": "poisson2d", "nodes": 271, "parts": 3, "mixed": True, "nrhs": 1, "reuse": False, "host": False},
        # the many-right-hand-sides workload: 261,121 unknowns, 32 columns at once, kept factors
        {"name": "poisson2d_513_mixed_rhs32", "kind": "poisson2d", "nodes": 513, "parts": 0, "mixed": True, "nrhs": 32, "reuse": True, "host": False},
        # a small 3-D system of odd size, FP64, ragged boxes
        {"name": "diffusion3d_45", "kind": "diffusion3d", "n": 45, "parts": 3, "mixed": False, "reuse": False},
        # time stepping: one more right-hand side of a matrix whose factors are kept
        {"name": "diffusion3d_64_mixed_reuse", "kind": "diffusion3d", "n": 64, "parts": 4, "mixed": True, "reuse": True},
        # a large plain FP64 solve
        {"name": "diffusion3d_96", "kind": "diffusion3d", "n": 96, "parts": 4, "mixed": False, "reuse": False},
        # the headline benchmark: 2,097,152 unknowns, 64 boxes, mixed precision
        {"name": "diffusion3d_128_mixed", "kind": "diffusion3d", "n": 128, "parts": 4, "mixed": True, "reuse": False},
        # many uneven independent systems in one call (the batched workload's lower half)
        {"name": "batch_48_mixed", "kind": "batch", "systems": 48, "n_max": 40000, "mixed": True},
        # elemental elasticity with the rigid-body coarse space
        {"name": "elasticity_26_mixed", "kind": "elasticity", "n": 26, "mixed": True},
        # one training step of a conductivity per element: forward, adjoint and gradients
        {"name": "adjoint_129_rhs8", "kind": "adjoint", "nodes": 129, "nrhs": 8},
        # the true residual of a solution a program already has
        {"name": "residual_128", "kind": "residual", "n": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["poisson2d", "poisson2d", "poisson2d", "diffusion3d", "diffusion3d", "diffusion3d", "batch",
                       "elasticity", "adjoint", "residual"])
    if kind == "poisson2d":
        nrhs = rng.choice([1, 1, _log(rng, 2, 32)])
        nodes = _log(rng, 25, 513)
        host = nrhs == 1 and rng.random() < 0.3
        return {"kind": kind, "nodes": nodes, "parts": 0 if nodes < 60 else rng.choice([0, 2, 3, 4]),
                "mixed": rng.random() < 0.5, "nrhs": nrhs, "reuse": rng.random() < 0.35, "host": host}
    if kind == "diffusion3d":
        mixed = rng.random() < 0.5
        n = _log(rng, 20, 120 if mixed else 96)
        return {"kind": kind, "n": n, "parts": max(2, min(4, round(n / 18))), "mixed": mixed, "reuse": rng.random() < 0.35}
    if kind == "batch":
        return {"kind": kind, "systems": _log(rng, 6, 64), "n_max": _log(rng, 6000, 40000), "mixed": rng.random() < 0.6}
    if kind == "elasticity":
        return {"kind": kind, "n": _log(rng, 8, 26), "mixed": rng.random() < 0.6}
    if kind == "adjoint":
        return {"kind": kind, "nodes": _log(rng, 33, 161), "nrhs": _log(rng, 1, 12)}
    return {"kind": kind, "n": _log(rng, 24, 128)}


# --- inputs ------------------------------------------------------------------
def _system(case, seed):
    """(n, rows1, cols1, vals, rhs columns, 1-based partition or None) of the assembled kinds."""
    if case["kind"] == "poisson2d":
        n, r, c, v, b, xy = P.poisson2d_p1(case["nodes"], seed=seed)
        k = case["parts"]
        part = None
        if k:
            box = np.minimum((xy * k).astype(int), k - 1)
            part = (1 + box[:, 0] * k + box[:, 1]).astype(np.int32)
        rng = np.random.default_rng(seed + 17)
        B = np.column_stack([b] + [rng.uniform(-1.0, 1.0, n) for _ in range(case["nrhs"] - 1)])
        return n, r, c, v, B, part
    n, r, c, v, b = P.diffusion3d_fv(case["n"], seed=seed)
    part = P.block_partition(case["n"], case["parts"]) if case["kind"] == "diffusion3d" else None
    return n, r, c, v, b[:, None], part


def _batch(case, seed):
    """(n, rows1, cols1, vals, rhs) of every system: sizes spread evenly over the logarithm of [2000, n_max], not in order."""
    k = case["systems"]
    sizes = np.exp(np.linspace(math.log(2000.0), math.log(case["n_max"]), k))[np.random.default_rng(k).permutation(k)]
    return [P.poisson2d_p1(int(round(math.sqrt(t))) + 2, seed=seed * 1009 + i)[:5] for i, t in enumerate(sizes)]


def _elasticity(case, seed):
    n = case["n"]
    ngf, eptr, efree, emat, erhs, info = P.elasticity3d_p1_elements(n, seed=seed)
    per = [max(2, min(k, round(n / 6))) for k in (4, 4, 8)]
    return ngf, eptr, efree, emat, erhs, info, P.dof_box_partition(info["node_ijk"], n, tuple(per))


def _adjoint(case, seed):
    rng = np.random.default_rng(seed + 4)
    ngf, eptr, efree, K, erhs, info = P.poisson2d_p1_elements(nodes=case["nodes"], seed=seed)
    kappa = np.exp(0.5 * rng.standard_normal(info["nell"]))
    B = rng.uniform(-1.0, 1.0, (ngf, case["nrhs"]))
    W = rng.uniform(-1.0, 1.0, (ngf, case["nrhs"]))  # the loss's gradient at the solution
    return ngf, eptr, efree, K, erhs, kappa, B, W


def _cuda(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "residual":
        n, r, c, v, b, _ = _system(case, seed)
        ptr = np.concatenate([[0], np.cumsum(np.bincount(r - 1, minlength=n))])
        x = np.random.default_rng(seed + 5).uniform(-1.0, 1.0, n)
        return {"kind": kind, "ptr": torch.tensor(ptr, dtype=torch.int64, device="cuda"),
                "col": torch.tensor(c - 1, dtype=torch.int32, device="cuda"), "val": _cuda(v), "x": _cuda(x), "b": _cuda(b[:, 0])}
    if kind == "adjoint":
        ngf, eptr, efree, K, erhs, kappa, B, W = _adjoint(case, seed)
        s = DougSolver(dict(CTLA, precision=1))
        return {"kind": kind, "solver": s, "mesh": (ngf, eptr, efree, K, erhs), "kappa": _cuda(kappa).requires_grad_(True),
                "B": _cuda(B).requires_grad_(True), "W": _cuda(W)}
    if kind == "batch":
        systems = _batch(case, seed)
        s = DougSolver(dict(CTL2, precision=int(case["mixed"])))
        s.set_systems([t[:4] for t in systems])
        b = np.concatenate([t[4] for t in systems])
        nrhs = 1
    elif kind == "elasticity":
        ngf, eptr, efree, emat, erhs, info, part = _elasticity(case, seed)
        s = DougSolver(dict(CTLE, precision=int(case["mixed"])))
        s.set_elements(ngf, eptr, efree, emat, erhs)
        s.set_node_geometry(info["coords"], info["freemap"])
        s.set_partition(part)
        b = s.input_matrix()[4]
        nrhs = 1
    else:
        n, r, c, v, B, part = _system(case, seed)
        s = DougSolver(dict(CTL3 if kind == "diffusion3d" else CTL2, precision=int(case["mixed"])))
        s.set_matrix_coo(n, r, c, v)
        if part is not None:
            s.set_partition(part)
        nrhs = B.shape[1]
        b = np.ascontiguousarray(B.T)
    if case.get("reuse"):
        s.set_option("reuse_factors", 1)
    s.setup()
    if case.get("host"):
        state = {"kind": "host", "solver": s, "b": b.reshape(-1)}
        if case.get("reuse"):
            s.solve(state["b"][::-1].copy())
        return state
    bd = _cuda(b).reshape(nrhs, -1)
    state = {"kind": "solve", "solver": s, "nrhs": nrhs, "b": bd, "x": torch.empty_like(bd)}
    if case.get("reuse"):  # the factors of an earlier solve, of another right-hand side
        _solve(state, bd.flip(1).contiguous())
    return state


def _solve(state, b):
    stream = torch.cuda.current_stream().cuda_stream
    if state["nrhs"] > 1:
        state["solver"].solve_multi_device(state["nrhs"], b.data_ptr(), state["x"].data_ptr(), stream)
    else:
        state["solver"].solve_device(b.data_ptr(), state["x"].data_ptr(), stream)
    return state["x"]


def run(state):
    kind = state["kind"]
    if kind == "solve":
        return _solve(state, state["b"])
    if kind == "host":
        return state["solver"].solve(state["b"])[0]
    if kind == "residual":
        return residual_csr(state["ptr"], state["col"], state["val"], state["x"], state["b"], torch.cuda.current_stream().cuda_stream)
    from doug_gb300.autograd import element_solve
    kappa, B = state["kappa"], state["B"]
    kappa.grad = B.grad = None
    X = element_solve(state["solver"], *state["mesh"], kappa, B)
    X.backward(state["W"])
    return X.detach(), kappa.grad, B.grad


def work(case):
    """Bytes: the matrix (8-byte values, 4-byte columns) and the right-hand
    sides read once, the solutions written once.  Flops: the products and
    vector updates of the PCG iterations at the counts these problems take to
    their tolerance; the preconditioner's are left out, being a choice of the
    method."""
    kind, sides, passes = case["kind"], case.get("nrhs", 1), 1
    if kind in ("poisson2d", "adjoint"):
        n = (case["nodes"] - 2) ** 2
        nnz, its = 7 * n, 40
        passes = 2 if kind == "adjoint" else 1
    elif kind == "batch":
        lo, hi = math.log(2000.0), math.log(case["n_max"])
        n = case["systems"] * (math.exp(hi) - math.exp(lo)) / (hi - lo)
        nnz, its = 7 * n, 40
    elif kind == "elasticity":
        n = 3 * case["n"] * (case["n"] + 1) ** 2
        nnz, its = 44 * n, 90
    else:
        n = case["n"] ** 3
        nnz, its = 7 * n, 50
    if kind == "residual":
        return {"bytes": 12.0 * nnz + 8.0 * (n + 1) + 24.0 * n + 8, "flops": 2.0 * nnz + 3.0 * n}
    return {"bytes": float(passes * (12 * nnz + 16 * n * sides)), "flops": float(passes * sides * its * (2 * nnz + 13 * n))}


# --- 64-bit values -------------------------------------------------------------
def _cg(A, B):
    """A X = B column by column with Jacobi-preconditioned CG in 64 bits, to rounding."""
    d = A["diag"][:, None]
    X = torch.zeros_like(B)
    Rm = B.clone()
    Z = Rm / d
    D = Z.clone()
    rz = (Rm * Z).sum(0)
    stop = 1e-30 * (B * B).sum(0)
    for it in range(30000):
        Q = A["csr"] @ D
        a = rz / (D * Q).sum(0).clamp_min(1e-300)
        X = X + a * D
        Rm = Rm - a * Q
        Z = Rm / d
        rz, old = (Rm * Z).sum(0), rz
        D = Z + (rz / old.clamp_min(1e-300)) * D
        if it % 100 == 99 and bool(((Rm * Rm).sum(0) <= stop).all()):
            break
    return X


def _csr(n, r, c, v):
    r, c, v = (torch.as_tensor(np.ascontiguousarray(t), device="cuda") for t in (r, c, v))
    A = torch.sparse_coo_tensor(torch.stack([r.long(), c.long()]), v.double(), (n, n)).coalesce()
    i, j = A.indices()
    diag = torch.zeros(n, dtype=torch.float64, device="cuda")
    diag[i[i == j]] = A.values()[i == j]
    return {"csr": A.to_sparse_csr(), "diag": diag}


def _assembled(n, eptr, efree, emat, scale=None):
    nf = np.diff(eptr)
    vals = emat if scale is None else emat * np.repeat(scale, nf * nf)
    e = np.repeat(np.arange(len(nf)), nf * nf)
    q = np.arange(len(emat)) - np.repeat(np.concatenate([[0], np.cumsum(nf * nf)])[:-1], nf * nf)
    i, j = q % nf[e], q // nf[e]
    return efree[eptr[e] + i] - 1, efree[eptr[e] + j] - 1, vals, e


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        systems = _batch(case, seed)
        off = np.concatenate([[0], np.cumsum([t[0] for t in systems])])
        r, c = (np.concatenate([t[k] - 1 + off[i] for i, t in enumerate(systems)]) for k in (1, 2))
        A = _csr(int(off[-1]), r, c, np.concatenate([t[3] for t in systems]))
        return _cg(A, _cuda(np.concatenate([t[4] for t in systems]))[:, None]).t().contiguous()
    if kind == "elasticity":
        ngf, eptr, efree, emat, erhs, _, _ = _elasticity(case, seed)
        i, j, v, _ = _assembled(ngf, eptr, efree, emat)
        b = np.bincount(efree - 1, weights=erhs, minlength=ngf)
        return _cg(_csr(ngf, i, j, v), _cuda(b)[:, None]).t().contiguous()
    if kind == "adjoint":
        ngf, eptr, efree, K, _, kappa, B, W = _adjoint(case, seed)
        i, j, v, e = _assembled(ngf, eptr, efree, K, kappa)
        A = _csr(ngf, i, j, v)
        X, L = _cg(A, _cuda(B)), _cg(A, _cuda(W))
        it, jt, et = (torch.as_tensor(t, device="cuda") for t in (i, j, e))
        g = torch.zeros(len(kappa), dtype=torch.float64, device="cuda")
        g.index_add_(0, et, -(L[it] * X[jt]).sum(1) * _cuda(K))
        return X, g, L
    n, r, c, v, B, _ = _system(case, seed)
    A = _csr(n, r - 1, c - 1, v)
    if kind == "residual":
        x = _cuda(np.random.default_rng(seed + 5).uniform(-1.0, 1.0, n))
        res = _cuda(B[:, 0]) - A["csr"] @ x
        return res, (res * res).sum().reshape(1)
    X = _cg(A, _cuda(B)).t().contiguous()
    return X.reshape(-1).cpu().numpy() if case.get("host") else X
