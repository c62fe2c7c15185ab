"""GPU: one subnormal pivot, at each position of an 8-column tile.

The tile factor takes a fast reciprocal square root that flushes subnormal
pivots and starts over with the library's when it met one; the last column of
a tile has no later pivot that could show it.  D = diag(1, ..., 1e-310, ..., 1)
factors exactly: sqrt of the stored value, ones elsewhere.  The square root of
a subnormal number is normal, so the bound is a few rounding errors.
Level nodes, and the block and warp workers of ragged batches.
"""
import numpy as np
import pytest
import torch

from socu_b200.block_tridiag_solver import calculate_off_diag_storage_len, create_cholesky_factor_launch
from socu_b200.ragged import RaggedBatch, create_ragged_factor_and_solve_launch

pytestmark = pytest.mark.gpu
TINY = 1e-310


def _blocks(N, n, pos):
    d = np.ones(n)
    d[pos] = TINY
    return np.stack([np.diag(d)] * N), np.zeros((calculate_off_diag_storage_len(N), n, n)), np.sqrt(d)


def _check(L, ref):
    got = torch.diagonal(L, dim1=-2, dim2=-1).cpu().numpy()
    assert np.abs(got / ref - 1.0).max() <= 4 * np.finfo(np.float64).eps
    assert not torch.tril(L, -1).any()


@pytest.mark.parametrize("n,pos", [(8, k) for k in range(8)] + [(1, 0), (7, 6), (20, 15), (24, 23), (64, 31), (72, 71),
                                                                 (128, 127)])
def test_level_node(n, pos):
    N = 3
    L0, E0, ref = _blocks(N, n, pos)
    L, E = torch.tensor(L0, device="cuda"), torch.tensor(E0, device="cuda")
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    create_cholesky_factor_launch(L, E, info=info)()
    torch.cuda.synchronize()
    assert info.tolist() == [0]
    _check(L, ref)


@pytest.mark.parametrize("copies", [1, 200])   # few nodes: block workers; more than 216 an SM: warp workers
def test_ragged_workers(copies):
    probs = [_blocks(256 if copies > 1 else 5, n, pos) for n, pos in [(8, 7), (16, 15), (20, 7), (24, 23), (8, 3)]]
    m = 1
    N = np.array([p[0].shape[0] for p in probs] * copies)
    n = np.array([p[0].shape[1] for p in probs] * copies)
    rb = RaggedBatch(N, n, np.full(N.shape, m), dtype=torch.float64)
    L, E, x = rb.empty()
    E.zero_()
    x.zero_()
    for i in range(rb.count):
        rb.L_view(L, i).copy_(torch.as_tensor(probs[i % len(probs)][0]))
    create_ragged_factor_and_solve_launch(rb, L, E, x)()
    torch.cuda.synchronize()
    assert rb.error_flag() == 0 and not x.any()
    for i in range(rb.count):
        _check(torch.tril(rb.L_view(L, i)), probs[i % len(probs)][2])


def test_reciprocal_root_over_the_exponent_range():
    """C = d r and F = r for 1x1 blocks, r = 1 / sqrt(d) by the approximate instruction and one
    third-order step.  The step leaves (5/16) e^3 < 2^-60 of the instruction's error and rounds
    d y (half of that reaches r) and r: 1.5 u; C adds a rounding, F at most the one of C and two more."""
    rng = np.random.default_rng(0)
    d = np.ldexp(1.0 + rng.random(40000), rng.integers(-1022, 1024, 40000))
    info = np.finfo(np.float64)
    d[:6] = [info.tiny, np.nextafter(info.tiny, 1.0), info.max, np.nextafter(info.max, 1.0), 1.0, np.nextafter(1.0, 0.0)]
    L = torch.ones(d.size, 2, 1, 1, dtype=torch.float64)
    L[:, 0, 0, 0] = torch.as_tensor(d)
    L, E = L.cuda(), torch.ones(d.size, 1, 1, 1, dtype=torch.float64, device="cuda")
    create_cholesky_factor_launch(L, E)()
    torch.cuda.synchronize()
    root = np.sqrt(d.astype(np.longdouble))
    u = np.longdouble(2.0) ** -53
    assert np.abs(L[:, 0, 0, 0].cpu().numpy() / root - 1).max() <= 2.5 * u
    assert np.abs(E[:, 0, 0, 0].cpu().numpy() * root - 1).max() <= 4.5 * u
