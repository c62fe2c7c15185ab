"""GPU: componentwise backward errors on ill-conditioned 8x8 diagonal tiles.

A triangular solve by substitution has a residual below (n + 3) u |C| |x| for
every C, a Cholesky factor one below (n + 1) u |C| |C^T| (Higham, Accuracy and
Stability of Numerical Algorithms, theorems 8.5 and 10.3), however
ill-conditioned C is; a product with an explicit inverse of a diagonal tile
does not: its residual grows with | |T^{-1}| |T| |.  Tiles here are bidiagonal,
I - a S, for which that number is about a^7 times the entries.  Right-hand
sides are C x with x of order one, so that the solves cancel.

Bounds: twice the theorems', with the rounding of a reciprocal pivot and of the
stored result (u each) added; the float kernels sum in FP64, so their error
does not grow past the eight columns of a tile.
"""
import numpy as np
import pytest
import torch

from socu_b200.block_tridiag_solver import (
    create_cholesky_backward_substitution_launch,
    create_cholesky_factor_launch,
    create_cholesky_forward_substitution_launch,
)
from socu_b200.ragged import RaggedBatch, create_ragged_factor_and_solve_launch

pytestmark = pytest.mark.gpu
ROUND = {torch.float64: 2.0 ** -53, torch.float32: 2.0 ** -24}
NP = {torch.float64: np.float64, torch.float32: np.float32}


def _bound(dtype, n):
    return 2 * ((n if dtype == torch.float64 else 8) + 8) * ROUND[dtype]


def _tile(n, a):
    return np.eye(n) - a * np.eye(n, k=-1)


def _ok(got, want, scale, bound):
    r = np.abs(got - want)
    assert (r <= bound * scale).all(), float((r[scale > 0] / scale[scale > 0]).max() / bound)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("m", [1, 8, 19])
@pytest.mark.parametrize("n", [5, 8, 29, 32, 64, 65, 100, 128])
def test_sweeps_on_a_plain_factor(dtype, n, m):
    rng = np.random.default_rng(n)
    C = np.tril(rng.standard_normal((n, n)) * 0.5 / np.sqrt(n), -1)
    for k in range(0, n, 8):
        e = min(n, k + 8)
        C[k:e, k:e] = _tile(e - k, 4.3)
    C = C.astype(NP[dtype])
    x0 = rng.standard_normal((n, m))
    E = torch.zeros(0, n, n, dtype=dtype, device="cuda")
    Cl = C.astype(np.longdouble)
    for make, M in ((create_cholesky_forward_substitution_launch, Cl), (create_cholesky_backward_substitution_launch, Cl.T)):
        b = (M @ x0).astype(NP[dtype])
        L, x = torch.tensor(C[None], device="cuda"), torch.tensor(b[None], device="cuda")
        make(L, E, x, dtype=dtype)()
        torch.cuda.synchronize()
        xl = x[0].cpu().numpy().astype(np.longdouble)
        _ok(M @ xl, b, np.abs(M) @ np.abs(xl), _bound(dtype, n))


def _spd(n, a, seed, np_dtype):
    """(L, E) of two blocks, L = C C^T with an ill-conditioned first tile in C_0, and E = F C_0^T."""
    rng = np.random.default_rng(seed)
    C = np.tril(rng.standard_normal((n, n)) * 0.5 / np.sqrt(n), -1) + np.eye(n)
    e = min(n, 8)
    C[:e, :e] = _tile(e, a)
    F = rng.standard_normal((n, n)) / np.sqrt(n)
    L = np.stack([C @ C.T, F @ F.T + 4.0 * np.eye(n)])
    return L.astype(np_dtype), (F @ C.T)[None].astype(np_dtype)


def _check_factor(L0, E0, L, E, dtype):
    n = L0.shape[1]
    C, F = np.tril(L[0]).astype(np.longdouble), E[0].astype(np.longdouble)
    _ok(np.tril(C @ C.T), np.tril(L0[0]), np.tril(np.abs(C) @ np.abs(C.T)), _bound(dtype, n))
    _ok(F @ C.T, E0[0], np.abs(F) @ np.abs(C.T), _bound(dtype, n))


GROWTH = {torch.float64: 3.3, torch.float32: 2.1}


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n", [8, 13, 16, 32, 64, 72, 100, 128])
def test_factor(dtype, n):
    L0, E0 = _spd(n, GROWTH[dtype], n, NP[dtype])
    L, E = torch.tensor(L0, device="cuda"), torch.tensor(E0, device="cuda")
    create_cholesky_factor_launch(L, E, dtype=dtype)()
    torch.cuda.synchronize()
    _check_factor(L0, E0, L.cpu().numpy(), E.cpu().numpy(), dtype)


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("copies", [1, 4200])   # block workers, warp workers
def test_ragged_factor(dtype, copies):
    probs = [_spd(n, GROWTH[dtype], n, NP[dtype]) for n in (8, 13, 16, 29)]
    count = len(probs) * copies
    n = np.array([p[0].shape[1] for p in probs] * copies)
    rb = RaggedBatch(np.full(count, 2), n, np.ones(count, dtype=np.int64), dtype=dtype)
    L = torch.tensor(np.concatenate([p[0].ravel() for p in probs]), device="cuda").repeat(copies)
    E = torch.tensor(np.concatenate([p[1].ravel() for p in probs]), device="cuda").repeat(copies)
    x = torch.zeros(rb.total_x, dtype=dtype, device="cuda")
    create_ragged_factor_and_solve_launch(rb, L, E, x)()
    torch.cuda.synchronize()
    assert rb.error_flag() == 0
    for i in list(range(len(probs))) + list(range(count - len(probs), count)):
        L0, E0 = probs[i % len(probs)]
        _check_factor(L0, E0, rb.L_view(L, i).cpu().numpy(), rb.E_view(E, i).cpu().numpy(), dtype)
