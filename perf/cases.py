"""The solve path's workloads as timed cases: what a user's program calls, at the sizes it calls it.

Grids and their Jacobians come from blockpowerflow_b200.grid (the benchmark's generator); the
topology of a case depends on its sizes alone and the operating point, the right-hand sides and
the network's weights on the seed, as a Newton or contingency loop meets one grid at many points.
A case's "kind" is the entry point it calls:

  mul     Y = A X, the CSR product of every Krylov step and residual check
  ldiv    ldiv_(Y, N, B): the ILU(0) triangular solves of every preconditioned step
  factor  N.refactor(values) and one vector solve: the preconditioner's part of a Newton step
  rf      update_(rf, A) and ldiv_(X, rf, B): the direct refactor + solve of a Newton step
  gmres   block_gmres with ILU(0) to 1e-8
  newton  newton(problem) with a kept RF solver, and the sensitivities to every control
  batch   BatchPlan.solve over independent grids, one graph launch
  mlp     loss and gradients of the learned warm start's network
"""
import dataclasses
import functools
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "blockpowerflow.jl_b200"))

import blockpowerflow_b200 as bpf  # noqa: E402
from blockpowerflow_b200 import grid as G  # noqa: E402
from blockpowerflow_b200 import learned as L  # noqa: E402
from blockpowerflow_b200 import newton as NT  # noqa: E402
from blockpowerflow_b200 import precond as P  # noqa: E402

RF = bpf.CUSOLVERRF
SIGMA = 0.01          # operating points: N(0, SIGMA) on every angle and magnitude
# The Newton cases move the point less: the larger grids have no solution, or several, close to some points.
POINT_SIGMA = 0.001
NEWTON_SIGMA = 0.0001  # how far a Newton loop starts from its solution


def listed():
    return [
        # one product on a 300-bus grid: nothing but launch and call latency
        {"name": "mul_300_p16", "kind": "mul", "n_bus": 300, "p": 16},
        # the product of the largest grid at the widest block: memory traffic
        {"name": "mul_70k_p128", "kind": "mul", "n_bus": 70000, "p": 128},
        # the preconditioner step of the 9,000-bus solve, in its minimum-degree order
        {"name": "ldiv_9k_p64_amd", "kind": "ldiv", "n_bus": 9000, "p": 64, "ordering": "AMD"},
        # the same at the largest grid, in the reference's natural order
        {"name": "ldiv_70k_p128", "kind": "ldiv", "n_bus": 70000, "p": 128, "ordering": "natural"},
        # new Jacobian values, ILU(0) again, one vector through it: an inexact Newton step
        {"name": "factor_9k", "kind": "factor", "n_bus": 9000},
        # a Newton step of a small grid: refactor and one right-hand side
        {"name": "rf_300_p1", "kind": "rf", "n_bus": 300, "p": 1},
        # a step of the refactorization sequence with a block of sensitivities
        {"name": "rf_25k_p256", "kind": "rf", "n_bus": 25000, "p": 256},
        # the reference's own solver test size, restarted
        {"name": "gmres_300_p16", "kind": "gmres", "n_bus": 300, "p": 16, "ordering": "natural", "memory": 30, "restart": True},
        # one whole unrestarted solve of a large grid
        {"name": "gmres_9k_p64", "kind": "gmres", "n_bus": 9000, "p": 64, "ordering": "AMD", "memory": 300, "restart": False},
        # the caller's loop: power flow and the sensitivities to all 1,001 controls
        {"name": "newton_9k", "kind": "newton", "n_bus": 9000},
        # half of the benchmark's batch: 256 grids of 100 - 3,000 buses, 8 - 64 right-hand sides each
        # (the whole one keeps 64 GB of basis blocks)
        {"name": "batch_256", "kind": "batch", "nsys": 256, "draw": 0},
        # one training batch of the learned warm start
        {"name": "mlp_9k_p64", "kind": "mlp", "n_bus": 9000, "p": 64, "hidden": 512},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["mul", "ldiv", "factor", "rf", "gmres", "newton", "batch", "mlp"])
    if kind in ("mul", "ldiv"):
        case = {"kind": kind, "n_bus": _log_int(rng, 300, 70000), "p": _log_int(rng, 1, 128)}
        if kind == "ldiv":
            case["ordering"] = rng.choice(["natural", "AMD"])
        return case
    if kind == "factor":
        return {"kind": kind, "n_bus": _log_int(rng, 300, 9000)}
    if kind == "rf":
        return {"kind": kind, "n_bus": _log_int(rng, 300, 25000), "p": _log_int(rng, 1, 256)}
    if kind == "gmres":
        # n / p >= 30: a block's Krylov space does not run out before the tolerance
        n_bus = _log_int(rng, 300, 9000)
        return {"kind": kind, "n_bus": n_bus, "p": _log_int(rng, 8, max(8, min(64, n_bus // 20))),
                "ordering": rng.choice(["natural", "AMD"]), "memory": 300, "restart": False}
    if kind == "newton":
        return {"kind": kind, "n_bus": _log_int(rng, 300, 9000)}
    if kind == "batch":
        return {"kind": kind, "nsys": _log_int(rng, 16, 256), "draw": rng.randrange(1, 1000)}
    return {"kind": "mlp", "n_bus": _log_int(rng, 300, 9000), "p": _log_int(rng, 1, 128), "hidden": rng.choice([128, 256, 512])}


# ---- inputs --------------------------------------------------------------------------------
PRESETS = dict(G.GRID_PRESETS.values())   # PV counts of the benchmark's own grids


@functools.lru_cache(maxsize=None)
def _problem(n_bus, topology):
    return NT.make_problem(G.make_grid(n_bus, PRESETS.get(n_bus) if topology == 0 else None, topology))


def _jacobian(n_bus, seed, topology=0):
    """(pattern, values, base values): the grid's Jacobian at a seeded operating point and at its own."""
    prob = _problem(n_bus, topology)
    g = prob.grid
    at = NT.perturbed_start(prob, SIGMA, seed)
    return prob.pattern, NT.jacobian_values(prob, at), NT.jacobian_values(prob, np.concatenate([g.va[1:], g.vm[g.pq]]))


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _gaussian(seed, rows, cols):
    """A seeded column-major rows x cols block of N(0, 1) values on the device."""
    gen = torch.Generator(device=_device()).manual_seed(seed)
    return torch.randn(cols, rows, dtype=torch.float64, device=_device(), generator=gen).t()


def _matrix(pattern, values):
    def ints(a):
        return torch.as_tensor(np.ascontiguousarray(a, dtype=np.int32), device="cuda")

    return bpf.CuSparseMatrixCSR(ints(pattern.indptr), ints(pattern.indices), torch.as_tensor(values, device="cuda"), pattern.shape[0])


def _batch_shapes(case):
    buses, nrhs = G.batch_sizes(case["nsys"], case["draw"])
    return buses, nrhs, [_problem(b, 1000 + k).pattern.shape[0] for k, b in enumerate(buses)]


def _batch_rhs(case, seed):
    """The right-hand sides of a batch: one flat buffer and its column-major block per system."""
    _, nrhs, n = _batch_shapes(case)
    flat = _gaussian(seed, sum(a * b for a, b in zip(n, nrhs)), 1).reshape(-1)
    return flat, _blocks(flat, n, nrhs)


def _blocks(flat, n, nrhs):
    out, at = [], 0
    for rows, cols in zip(n, nrhs):
        out.append(flat[at:at + rows * cols].view(cols, rows).t())
        at += rows * cols
    return out


def _newton_problem(case, seed):
    """The grid at a seeded operating point, which is the power flow's solution."""
    base = _problem(case["n_bus"], 0).grid
    rng = np.random.default_rng(seed)
    va = base.va + rng.normal(0.0, POINT_SIGMA, base.n_bus)
    va[0] = 0.0
    return NT.make_problem(dataclasses.replace(base, vm=base.vm + rng.normal(0.0, POINT_SIGMA, base.n_bus), va=va))


def _weights(case, n, seed):
    """The network's parameters (LeCun-normal weights, small biases), padding zero."""
    gen = torch.Generator(device=_device()).manual_seed(seed + 1)
    h, npad = case["hidden"], -(-n // 128) * 128

    def normal(rows, cols, scale, valid_rows, valid_cols):
        w = torch.randn(rows, cols, device=_device(), generator=gen) * scale
        w[valid_rows:] = 0
        w[:, valid_cols:] = 0
        return w

    return {"W1": normal(h, npad, n ** -0.5, h, n), "b1": normal(1, h, 0.01, 1, h), "W2": normal(h, h, h ** -0.5, h, h),
            "b2": normal(1, h, 0.01, 1, h), "W3": normal(npad, h, h ** -0.5, n, h), "b3": normal(1, npad, 0.01, 1, n)}


def _pairs(case, seed):
    """(B, X) with A X = B for a training batch, and the set's median ||x|| / ||b||."""
    pattern, values, _ = _jacobian(case["n_bus"], seed)
    X = _gaussian(seed, pattern.shape[0], case["p"])
    B = _product(pattern, values, X)
    return B, X, float((X.norm(dim=0) / B.norm(dim=0)).median())


def _product(pattern, values, X):
    """A X in 64 bits by torch alone (column-major)."""
    rows = torch.as_tensor(np.repeat(np.arange(pattern.shape[0]), np.diff(pattern.indptr)), device=X.device)
    cols = torch.as_tensor(pattern.indices.astype(np.int64), device=X.device)
    vals = torch.as_tensor(values, device=X.device)
    Y = torch.zeros(X.shape[1], X.shape[0], dtype=torch.float64, device=X.device)
    for j in range(X.shape[1]):
        Y[j].index_add_(0, rows, vals * X[:, j][cols])
    return Y.t()


# ---- the cases -----------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        buses, nrhs, n = _batch_shapes(case)
        mats = []
        for k, b in enumerate(buses):
            prob = _problem(b, 1000 + k)
            mats.append(_matrix(prob.pattern, NT.jacobian_values(prob, NT.perturbed_start(prob, SIGMA, seed + k))))
        _, B = _batch_rhs(case, seed)
        flat = torch.zeros(sum(a * b for a, b in zip(n, nrhs)), dtype=torch.float64, device="cuda")
        # slice width and order as the autotuner picks them for this batch
        plan = bpf.BatchPlan(mats, nrhs, rtol=1e-8, slice=32, ordering="RCM")
        return {"kind": kind, "plan": plan, "B": B, "X": _blocks(flat, n, nrhs), "flat": flat}
    if kind == "newton":
        prob = _newton_problem(case, seed)
        return {"kind": kind, "prob": prob, "x0": NT.perturbed_start(prob, NEWTON_SIGMA, seed),
                "solver": NT.RFSolver(prob, len(prob.ctrl))}
    if kind == "mlp":
        B, X, scale = _pairs(case, seed)
        net = L.WarmStartMLP(X.shape[0], case["hidden"], seed=0)
        net.set_scale(scale)
        for name, w in _weights(case, X.shape[0], seed).items():
            net.set_param(name, w)
        return {"kind": kind, "net": net, "B": B, "X": X}
    pattern, values, base = _jacobian(case["n_bus"], seed)
    A = _matrix(pattern, values)
    state = {"kind": kind, "A": A, "B": _gaussian(seed, A.n, case.get("p", 1))}
    if kind == "ldiv":
        state["N"] = bpf.ilu0(A, case["p"], ordering=case["ordering"])
    if kind == "factor":
        state["N"] = bpf.ilu0(_matrix(pattern, base), 1)
        state["B"] = state["B"][:, 0]
    if kind == "rf":
        state["rf"] = RF.CusolverRfLU(_matrix(pattern, base), nrhs=case["p"])
    if kind == "gmres":
        state["N"] = bpf.ilu0(A, case["p"], ordering=case["ordering"])
        state["memory"], state["restart"] = case["memory"], case["restart"]
    if kind in ("ldiv", "rf"):
        state["X"] = bpf.empty_colmajor(A.n, case["p"])
    return state


def run(s):
    kind = s["kind"]
    if kind == "mul":
        return bpf.mul(s["A"], s["B"])
    if kind == "ldiv":
        return P.ldiv_(s["X"], s["N"], s["B"])
    if kind == "factor":
        s["N"].refactor(s["A"].nzVal)
        return {"factors": s["N"].P.nzVal, "y": s["N"].ldiv(s["B"])}
    if kind == "rf":
        RF.update_(s["rf"], s["A"])
        return RF.ldiv_(s["X"], s["rf"], s["B"])
    if kind == "gmres":
        X, _ = bpf.block_gmres(s["A"], s["B"], N=s["N"], ldiv=True, restart=s["restart"], memory=s["memory"], atol=0.0,
                               rtol=1e-8, itmax=300)
        return X
    if kind == "newton":
        r = NT.newton(s["prob"], solver=s["solver"], x0=s["x0"], sensitivities=True)
        return {"x": r.x, "vm": r.vm, "va": r.va, "sensitivities": r.sensitivities}
    if kind == "batch":
        s["plan"].solve(s["B"], s["X"])
        return s["flat"]
    loss = s["net"].gradients(s["B"], s["X"])
    return {"loss": loss, **{name: s["net"].param(name, grad=True) for name in L.PARAMS}}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        _, nrhs, n = _batch_shapes(case)
        parts = [_gmres_work(a, 7 * a, b, min(32, b)) for a, b in zip(n, nrhs)]
        return {"bytes": sum(x["bytes"] for x in parts), "flops": sum(x["flops"] for x in parts)}
    if kind == "mlp":
        n, p, h = _problem(case["n_bus"], 0).pattern.shape[0], case["p"], case["hidden"]
        weights = 2 * n * h + h * h
        return {"bytes": 16 * n * p + 2 * weights + 4 * weights, "flops": 2 * p * (3 * weights - n * h)}
    pattern = _problem(case["n_bus"], 0).pattern
    n, nnz, p = pattern.shape[0], pattern.nnz, case.get("p", 1)
    if kind == "newton":
        # the Jacobian's values and pattern, and the dense n x controls block, in and out
        c = _problem(case["n_bus"], 0).grid.n_bus * 2 - 1 - n + 1
        return {"bytes": 12 * nnz + 16 * n * c, "flops": 4 * nnz * c}
    if kind == "gmres":
        return _gmres_work(n, nnz, p, p)
    # pattern and values in, block in, block out (factor: the new factors out as well)
    extra = 8 * nnz if kind == "factor" else 0
    return {"bytes": 12 * nnz + 4 * (n + 1) + 16 * n * p + extra, "flops": 2 * nnz * p}


def _gmres_work(n, nnz, p, width):
    """Matrix and blocks in and out; one Gram-Schmidt pass, a product and a preconditioner solve per
    iteration, with the iteration count these grids' ILU(0) takes, 1.5 (n / width)^0.7."""
    k = 1.5 * (n / width) ** 0.7
    return {"bytes": 12 * nnz + 16 * n * p, "flops": 2 * n * p * width * k * k + 4 * nnz * p * k}


# ---- the same outputs in 64 bits, by torch and numpy ------------------------------------------
def _dense(pattern, values):
    n = pattern.shape[0]
    A = torch.zeros(n, n, dtype=torch.float64, device=_device())
    rows = torch.as_tensor(np.repeat(np.arange(n), np.diff(pattern.indptr)), device=A.device)
    A[rows, torch.as_tensor(pattern.indices.astype(np.int64), device=A.device)] = torch.as_tensor(values, device=A.device)
    return A


def _ilu0(pattern, values):
    """ILU(0) on the pattern, row by row: the combined factors in the pattern's order."""
    ptr, col, v = pattern.indptr.tolist(), pattern.indices.tolist(), values.tolist()
    diag = [0] * pattern.shape[0]
    for i in range(pattern.shape[0]):
        at = {col[q]: q for q in range(ptr[i], ptr[i + 1])}
        diag[i] = at[i]
        for q in range(ptr[i], at[i]):
            k = col[q]
            v[q] /= v[diag[k]]
            for r in range(diag[k] + 1, ptr[k + 1]):
                if col[r] in at:
                    v[at[col[r]]] -= v[q] * v[r]
    return np.array(v), np.array(diag)


def _ilu0_solve(pattern, v, diag, B):
    y = np.array(B)
    ptr, col = pattern.indptr, pattern.indices
    for i in range(len(y)):
        a, d = ptr[i], diag[i]
        if d > a:
            y[i] -= v[a:d] @ y[col[a:d]]
    for i in range(len(y) - 1, -1, -1):
        d, e = diag[i], ptr[i + 1]
        if e > d + 1:
            y[i] -= v[d + 1:e] @ y[col[d + 1:e]]
        y[i] /= v[d]
    return y


def _newton_exact(case, seed):
    """The power flow's solution is the grid's own operating point; dx/du = -Gx^-1 Gu there, from
    dS/dtheta = j V (conj(I) - conj(Y V)) and dS/d|V| = V conj(Y V/|V|) + conj(I) V/|V|."""
    prob = _newton_problem(case, seed)
    g, dev = prob.grid, _device()
    y = torch.as_tensor(1.0 / (g.r + 1j * g.x), device=dev)
    f, t = torch.as_tensor(g.f, device=dev), torch.as_tensor(g.t, device=dev)
    Y = torch.zeros(g.n_bus, g.n_bus, dtype=torch.complex128, device=dev)
    for a, b, v in ((f, t, -y), (t, f, -y), (f, f, y), (t, t, y)):
        Y.index_put_((a, b), v, accumulate=True)
    V = torch.as_tensor(g.vm * np.exp(1j * g.va), device=dev)
    Vn, I = V / V.abs(), Y @ V
    dth = 1j * (torch.diag(V * I.conj()) - V[:, None] * (Y * V).conj())
    dvm = V[:, None] * (Y * Vn).conj() + torch.diag(I.conj() * Vn)
    pq, ctrl = torch.as_tensor(g.pq, device=dev), torch.as_tensor(prob.ctrl, device=dev)
    del Y
    Gx = torch.cat([torch.cat([dth[1:, 1:].real, dvm[1:][:, pq].real], 1), torch.cat([dth[pq, 1:].imag, dvm[pq][:, pq].imag], 1)])
    Gu = torch.cat([dvm[1:][:, ctrl].real, dvm[pq][:, ctrl].imag])
    return {"x": np.concatenate([g.va[1:], g.vm[g.pq]]), "vm": g.vm, "va": g.va, "sensitivities": -torch.linalg.solve(Gx, Gu)}


def _mlp_exact(case, seed):
    """The network's loss and gradients without any rounding to 16 bits."""
    B, X, scale = _pairs(case, seed)
    n, p = X.shape
    w = {k: v.double().requires_grad_() for k, v in _weights(case, n, seed).items()}
    bn = B.norm(dim=0)
    u = torch.nn.functional.pad((B / bn).t(), (0, w["W1"].shape[1] - n))
    a = torch.nn.functional.leaky_relu(u @ w["W1"].t() + w["b1"], 0.25)
    a = torch.nn.functional.leaky_relu(a @ w["W2"].t() + w["b2"], 0.25)
    y = (a @ w["W3"].t() + w["b3"])[:, :n]
    t = (X / (scale * bn)).t()
    loss = ((y - t).square().sum(1) / t.square().sum(1)).mean()
    grads = torch.autograd.grad(loss, [w[k] for k in L.PARAMS])
    return {"loss": float(loss), **dict(zip(L.PARAMS, grads))}


def exact(case, seed):
    kind = case["kind"]
    if kind == "newton":
        return _newton_exact(case, seed)
    if kind == "mlp":
        return _mlp_exact(case, seed)
    if kind == "batch":
        _, B = _batch_rhs(case, seed)
        out = []
        for k, b in enumerate(_batch_shapes(case)[0]):
            prob = _problem(b, 1000 + k)
            A = _dense(prob.pattern, NT.jacobian_values(prob, NT.perturbed_start(prob, SIGMA, seed + k)))
            out.append(torch.linalg.solve(A, B[k]).t().reshape(-1))
        return torch.cat(out)
    pattern, values, _ = _jacobian(case["n_bus"], seed)
    B = _gaussian(seed, pattern.shape[0], case.get("p", 1))
    if kind == "mul":
        return _product(pattern, values, B)
    if kind == "factor" or (kind == "ldiv" and case["ordering"] == "natural"):
        v, diag = _ilu0(pattern, values)
        y = _ilu0_solve(pattern, v, diag, B.cpu().numpy())
        return y if kind == "ldiv" else {"factors": v, "y": y[:, 0]}
    if kind in ("rf", "gmres") and pattern.shape[0] <= 20000:
        return torch.linalg.solve(_dense(pattern, values), B)
    return None   # the factors' order is the library's own, or the dense solve takes too long
