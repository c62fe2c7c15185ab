"""The solver's work as its users run it: the cases, their inputs and one pass of each.

Every case goes through a public entry point: the launch factories of
``socu_b200.block_tridiag_solver`` (bound once, called per solve, as the
reference's callers do), the refined solve, the ragged batches and the
differentiable solve.  Inputs are the README construction (block-bidiagonal
C with random blocks, Psi = C C^T) with a diagonal shift of 10 + 2 sqrt(n),
for which Psi is positive definite at every block size used here.

The factor entry points work in place, so a pass first copies the step's
inputs into the bound buffers, as a control loop does with each new problem.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from socu_b200.autograd import block_tridiag_solve
from socu_b200.block_tridiag_solver import (
    calculate_off_diag_storage_len,
    calculate_recursive_iterations,
    create_cholesky_factor_and_solve_launch,
    create_cholesky_factor_launch,
    create_cholesky_solve_launch,
)
from socu_b200.mixed import create_cholesky_refined_solve_launch
from socu_b200.problems import fill_ragged, ragged_shapes, readme_blocks
from socu_b200.ragged import (
    RaggedBatch,
    create_ragged_factor_and_solve_launch,
    create_ragged_refined_solve_launch,
)

DEVICE = "cuda"

# cost limits of a drawn case: floating-point operations and block elements of
# one pass, below the largest listed cases
MAX_FLOPS = 2.0e10
MAX_ELEMS = 6.0e7


def _uniform(name, op, B, N, n, m, dtype="f64", graph=True, inverse=False, mask=False):
    return {"name": name, "op": op, "B": B, "N": N, "n": n, "m": m, "dtype": dtype, "graph": graph,
            "inverse": inverse, "mask": mask}


def _ragged(name, count, seed, refine):
    return {"name": name, "op": "ragged", "count": count, "shapes_seed": seed, "refine": refine}


def listed():
    return [
        # a small controller's problem, the factory's defaults (no CUDA graph): latency and launches
        _uniform("fs_f64_N20_n10_eager", "factor_and_solve", 1, 20, 10, 1, graph=False),
        # the README's single system
        _uniform("fs_f64_N100_n32_m1", "factor_and_solve", 1, 100, 32, 1),
        # float32, a block size that is no power of two, one system
        _uniform("fs_f32_N100_n36_m1", "factor_and_solve", 1, 100, 36, 1, dtype="f32"),
        # the headline system in plain FP64
        _uniform("fs_f64_N1024_n64_m8", "factor_and_solve", 1, 1024, 64, 8),
        # the headline system: float factor with FP64 refinement
        _uniform("refined_N1024_n64_m8", "refined", 1, 1024, 64, 8),
        # a batch of odd-sized systems, some switched off by the mask; factor and solve as two calls, eager
        _uniform("factor_solve_f64_B24_N63_n17_m3", "factor+solve", 24, 63, 17, 3, graph=False, mask=True),
        # many right-hand sides in turn on one stored factor that kept its inverses, float32
        _uniform("solve_f32_inv_N1024_n64_m8", "solve", 1, 1024, 64, 8, dtype="f32", inverse=True),
        # a batch of stored FP64 factors without inverses (the reference's factor format)
        _uniform("solve_f64_B32_N128_n32_m4", "solve", 32, 128, 32, 4),
        # large blocks, many right-hand sides: the compute-bound end
        _uniform("fs_f64_N2048_n128_m32", "factor_and_solve", 1, 2048, 128, 32),
        # uneven MPC-style batch, plain FP64
        _ragged("ragged_f64_1024", 1024, 0, False),
        # the same kind of batch, float factor with FP64 refinement
        _ragged("ragged_refined_512", 512, 5000, True),
        # differentiable solve: forward and backward of a batch of short systems
        _uniform("autograd_f64_B256_N128_n16_m1", "autograd", 256, 128, 16, 1),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["factor_and_solve", "factor_and_solve", "refined", "factor+solve", "solve", "ragged", "autograd"])
    if op == "ragged":
        return {"op": op, "count": _log_int(rng, 16, 512), "shapes_seed": rng.randrange(1 << 20),
                "refine": rng.random() < 0.4}
    while True:
        B, N = _log_int(rng, 1, 256), _log_int(rng, 4, 4096)
        n, m = _log_int(rng, 4, 128), _log_int(rng, 1, 32)
        case = {"op": op, "B": B, "N": N, "n": n, "m": m, "dtype": rng.choice(["f64", "f64", "f32"]),
                "graph": rng.random() < 0.6, "inverse": n <= 64 and rng.random() < 0.5,
                "mask": B > 1 and rng.random() < 0.3}
        if op in ("refined", "autograd"):
            case.update(dtype="f64", graph=True, inverse=False, mask=False)
        if work(case)["flops"] <= MAX_FLOPS and B * 3 * N * n * n <= MAX_ELEMS:
            return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _shift(n):
    return 10.0 + 2.0 * math.sqrt(n)


def _ragged_shapes(case):
    return ragged_shapes(case["shapes_seed"], case["count"])


def _inputs(case, seed):
    """(L, E, b) of a case in FP64: uniform arrays, or the packed arrays of a ragged batch."""
    if case["op"] == "ragged":
        batch = _batch(case)
        L, E, b = batch.empty()
        fill_ragged(batch, L, E, b, seed=7919 * seed, shift=_shift(48))
        return L, E, b
    return readme_blocks(case["N"], case["n"], case["m"], shift=_shift(case["n"]), seed=seed, batch=case["B"],
                         device=DEVICE)


def _batch(case):
    N, n, m = _ragged_shapes(case)
    return RaggedBatch(N, n, m, dtype=torch.float64, device=DEVICE, refine=case["refine"])


def _mask(case):
    """Every third entry of a masked batch is switched off."""
    if not case["mask"]:
        return None
    return (torch.arange(case["B"], device=DEVICE) % 3 != 1)


def prepare(case, seed):
    op = case["op"]
    L0, E0, b0 = _inputs(case, seed)
    s = {"op": op}
    if op == "ragged":
        s["batch"] = batch = _batch(case)
        if case["refine"]:
            s["x"] = torch.zeros_like(b0)
            s["launch"] = create_ragged_refined_solve_launch(batch, L0, E0, b0, s["x"])
            return s
        s["in"] = (L0, E0, b0)
        s["work"] = tuple(a.clone() for a in s["in"])
        s["launch"] = create_ragged_factor_and_solve_launch(batch, *s["work"])
        return s
    if op == "refined":
        s["x"] = torch.zeros_like(b0)
        s["launch"] = create_cholesky_refined_solve_launch(L0, E0, b0, s["x"], use_cuda_graph=case["graph"])
        return s
    if op == "autograd":
        D, E, b = L0, E0[:, :case["N"] - 1].contiguous(), b0
        s["in"] = tuple(a.requires_grad_(True) for a in (D, E, b))
        g = torch.Generator(device=DEVICE).manual_seed(seed + 1)
        s["w"] = torch.randn(b.shape, generator=g, device=DEVICE, dtype=torch.float64)
        return s
    dt = torch.float32 if case["dtype"] == "f32" else torch.float64
    s["in"] = tuple(a.to(dt) for a in (L0, E0, b0))
    s["work"] = L, E, x = tuple(a.clone() for a in s["in"])
    mask = _mask(case)
    kw = dict(mask=mask, dtype=dt, use_cuda_graph=case["graph"])
    if op == "factor_and_solve":
        s["launch"] = create_cholesky_factor_and_solve_launch(L, E, x, **kw)
        return s
    s["factor"] = create_cholesky_factor_launch(L, E, keep_inverse=case["inverse"], **kw)
    s["solve"] = create_cholesky_solve_launch(L, E, x, factor_has_inverse=case["inverse"], **kw)
    if op == "solve":
        s["factor"]()
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

def run(state):
    op = state["op"]
    if op == "autograd":
        D, E, b = state["in"]
        x = block_tridiag_solve(D, E, b)
        gD, gE, gb = torch.autograd.grad(x, (D, E, b), state["w"])
        return {"x": x, "dD": gD, "dE": gE, "db": gb}
    if "work" not in state:   # refined solves leave their inputs as they are
        state["launch"]()
        return {"x": state["x"]}
    L, E, x = state["work"]
    if op != "solve":
        L.copy_(state["in"][0])
        E.copy_(state["in"][1])
    x.copy_(state["in"][2])
    if "launch" in state:
        state["launch"]()
    else:
        if op == "factor+solve":
            state["factor"]()
        state["solve"]()
    return {"x": x} if op == "solve" else {"L": L, "E": E, "x": x}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _factor_flops(N, n):
    """Per node: Cholesky n^3/3, two triangular block solves of n^3, two
    symmetric rank-n updates of n^3 and one fill-in product of 2 n^3."""
    return N * n ** 3 * (1.0 / 3.0 + 6.0)


def _sweep_flops(N, n, m):
    """Forward and backward sweep: a triangular solve and two block products each."""
    return 2.0 * N * n * n * m * (1.0 + 4.0)


def work(case):
    op = case["op"]
    if op == "ragged":
        flops = byts = 0.0
        for N, n, m in zip(*(a.tolist() for a in _ragged_shapes(case))):
            S = calculate_off_diag_storage_len(N)
            flops += _factor_flops(N, n) + _sweep_flops(N, n, m)
            if case["refine"]:   # blocks read once, b read, x written
                flops += _sweep_flops(N, n, m)
                byts += 8.0 * ((2 * N - 1) * n * n + 2 * N * n * m)
            else:
                byts += 8.0 * (2 * (N + S) * n * n + 2 * N * n * m)
        return {"bytes": byts, "flops": flops}
    B, N, n, m = case["B"], case["N"], case["n"], case["m"]
    S = calculate_off_diag_storage_len(N)
    w = 4.0 if case["dtype"] == "f32" else 8.0
    blocks, vec = (N + S) * n * n * w, N * n * m * w
    factor, sweep = _factor_flops(N, n), _sweep_flops(N, n, m)
    if op == "solve":
        byts, flops = blocks + 2 * vec, sweep
    elif op == "refined":   # one correction at least: a second sweep pair and an FP64 residual
        byts, flops = (2 * N - 1) * n * n * w + 2 * vec, factor + 2 * sweep + 6.0 * N * n * n * m
    elif op == "autograd":   # factor, two solves, two outer products per row; D, E, b, w in, x and gradients out
        byts = 2 * (2 * N - 1) * n * n * w + 4 * vec
        flops = factor + 2 * sweep + 6.0 * N * n * n * m
    else:
        byts, flops = 2 * blocks + 2 * vec, factor + sweep
    return {"bytes": B * byts, "flops": B * flops}


# ---------------------------------------------------------------------------
# the same results from plain torch in 64 bits
# ---------------------------------------------------------------------------

def _nested_dissection(L, E, x, inverse):
    """In-place factor of (L, E) and solution of x (batch first), one separator level at a time.

    lower(L_i) = C_i with zeros above, or W_i^T = C_i^{-T} above when `inverse`."""
    N, n = L.shape[1], L.shape[2]
    eye = torch.eye(n, dtype=L.dtype, device=L.device)
    levels, s, cur, nxt = [], 1, 0, N - 1

    def lower(C, V):
        return torch.linalg.solve_triangular(C, V, upper=False)

    for _ in range(calculate_recursive_iterations(N)):
        d = (N + s) // (2 * s)
        node = torch.arange(d, device=L.device) * (2 * s) + s - 1
        low = torch.tril(L[:, node])
        C = torch.linalg.cholesky(low + torch.tril(low, -1).transpose(-1, -2))
        right = int((node + s < N).sum())   # only the last node may lack a right neighbour
        if right:
            slots = cur + 2 * torch.arange(right, device=L.device)
            E[:, slots] = lower(C[:, :right], E[:, slots].transpose(-1, -2)).transpose(-1, -2)
        if d > 1:
            slots = cur + 2 * torch.arange(1, d, device=L.device) - 1
            E[:, slots] = lower(C[:, 1:], E[:, slots])
        x[:, node] = lower(C, x[:, node])
        L[:, node] = C
        if inverse:
            L[:, node] += torch.triu(lower(C, eye.expand_as(C)).transpose(-1, -2), 1)
        levels.append((s, cur, d, right, node, C))
        U = N // (2 * s)
        if U:
            u = torch.arange(1, U + 1, device=L.device)
            j = 2 * s * u - 1
            F = E[:, cur + 2 * (u - 1)]
            L[:, j] -= F @ F.transpose(-1, -2)
            x[:, j] -= F @ x[:, j - s]
            u, j = u[j + s < N], j[j + s < N]
            G = E[:, cur + 2 * u - 1]
            L[:, j] -= G.transpose(-1, -2) @ G
            x[:, j] -= G.transpose(-1, -2) @ x[:, j + s]
        if right > 1:   # nodes with two neighbours
            both = torch.arange(1, right, device=L.device)
            E[:, nxt + both - 1] -= E[:, cur + 2 * both] @ E[:, cur + 2 * both - 1]
        s, cur = 2 * s, nxt
        nxt += N // s - 1
    for s, cur, d, right, node, C in reversed(levels):
        y = x[:, node]
        if right:
            F = E[:, cur + 2 * torch.arange(right, device=L.device)]
            y[:, :right] -= F.transpose(-1, -2) @ x[:, node[:right] + s]
        if d > 1:
            G = E[:, cur + 2 * torch.arange(1, d, device=L.device) - 1]
            y[:, 1:] -= G @ x[:, node[1:] - s]
        x[:, node] = torch.linalg.solve_triangular(C.transpose(-1, -2), y, upper=True)


def exact(case, seed):
    op = case["op"]
    L, E, b = _inputs(case, seed)
    if op == "ragged":
        batch = _batch(case)
        x = b.clone()
        for i in range(batch.count):
            _nested_dissection(batch.L_view(L, i)[None], batch.E_view(E, i)[None], batch.x_view(x, i)[None], True)
        return {"x": x} if case["refine"] else {"L": L, "E": E, "x": x}
    if op == "autograd":
        N = case["N"]
        x = b.clone()
        _nested_dissection(L, E, x, False)
        L, E, _ = _inputs(case, seed)
        g = torch.Generator(device=DEVICE).manual_seed(seed + 1)
        gb = torch.randn(b.shape, generator=g, device=DEVICE, dtype=torch.float64)
        _nested_dissection(L, E, gb, False)
        full = -(gb @ x.transpose(-1, -2))
        dD = torch.tril(full, -1) + torch.tril(full.transpose(-1, -2), -1) + torch.diag_embed(
            full.diagonal(dim1=-2, dim2=-1))
        dE = -(gb[:, 1:] @ x[:, :N - 1].transpose(-1, -2) + x[:, 1:] @ gb[:, :N - 1].transpose(-1, -2))
        return {"x": x, "dD": dD, "dE": dE, "db": gb}
    if case["dtype"] == "f32":   # the inputs that the float run is given
        L, E, b = (a.float().double() for a in (L, E, b))
    mask = _mask(case)
    L0, E0, b0 = (a.clone() for a in (L, E, b)) if mask is not None else (None, None, None)
    x = b
    _nested_dissection(L, E, x, op == "factor_and_solve" and case["n"] <= 64 or case["inverse"])
    if mask is not None:
        for a, a0 in ((L, L0), (E, E0), (x, b0)):
            a[~mask] = a0[~mask]
    return {"x": x} if op in ("solve", "refined") else {"L": L, "E": E, "x": x}
