"""GPU: the level node that keeps its row tiles in registers (n <= 128).

Factor blocks, inverses and solutions against the oracle at the edges of its
8-column tiles (one short of, at and past a tile; even and odd tile counts),
for blocks that start off a 16-byte boundary, and on narrow levels (a cluster
of thread blocks per node) against wide ones (one block per node), which must
agree bit for bit.  Bounds: the backward-stable n * eps growth of a blocked
Cholesky on these well-conditioned blocks, n * eps <= 3e-14 (FP64) and 1.6e-5
(float) at n = 128, with a margin of 30 and 6.
"""
import numpy as np
import pytest
import torch

from oracle import generators, nd_cholesky as nd
from socu_b200.block_tridiag_solver import (
    calculate_off_diag_storage_len,
    create_cholesky_factor_and_solve_launch,
    create_cholesky_factor_launch,
)

pytestmark = pytest.mark.gpu
REL = {torch.float64: 1e-12, torch.float32: 1e-4}


def _problem(N, n, m, seed):
    return generators.readme_problem(N, n, m, shift=10.0 + 2.0 * np.sqrt(n), seed=seed)


def _dev(a, dtype, offset=0):
    """A contiguous device copy whose storage starts `offset` elements into an allocation."""
    t = torch.empty(a.size + offset, dtype=dtype, device="cuda")
    v = t[offset:].view(a.shape)
    v.copy_(torch.as_tensor(a))
    return v


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n,m,offset", [(1, 1, 0), (7, 2, 0), (8, 9, 1), (9, 1, 0), (16, 1, 0), (25, 3, 0),
                                        (39, 8, 0), (48, 4, 1), (56, 17, 0), (63, 1, 0), (64, 33, 0), (65, 2, 0),
                                        (72, 5, 0), (88, 1, 0), (97, 8, 0), (104, 3, 1), (120, 1, 0), (127, 2, 0),
                                        (128, 9, 0)])
def test_factor_and_solution_match_oracle(dtype, n, m, offset):
    N = 13
    L0, E0, b0 = _problem(N, n, m, n)
    Lr, Er, xr = (a[0] for a in nd.nd_factor_and_solve(L0, E0, b0))
    L, E, x = (_dev(a, dtype, offset) for a in (L0, E0, b0))
    create_cholesky_factor_and_solve_launch(L, E, x, dtype=dtype)()
    torch.cuda.synchronize()
    tol = REL[dtype]
    Lg = L.double().cpu().numpy()
    for got, ref in ((np.tril(Lg), np.tril(Lr)), (E.double().cpu().numpy(), Er), (x.double().cpu().numpy(), xr)):
        assert np.abs(got - ref).max() <= tol * np.abs(ref).max()
    if n <= 64:   # the strict upper triangles carry C^{-T}
        inv = np.triu(np.linalg.inv(np.tril(Lr)).transpose(0, 2, 1), 1)
        assert np.abs(np.triu(Lg, 1) - inv).max() <= tol * max(1.0, np.abs(inv).max())
    # factor alone: zeros above the diagonal, the same bits below
    L2, E2 = (_dev(a, dtype, offset) for a in (L0, E0))
    create_cholesky_factor_launch(L2, E2, dtype=dtype)()
    torch.cuda.synchronize()
    assert torch.equal(torch.tril(L2), torch.tril(L)) and torch.equal(E2, E)
    assert not torch.triu(L2, 1).any()


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n", [12, 64, 100])
def test_clusters_and_single_blocks_agree_bitwise(dtype, n):
    N, m, B = 6, 2, 120
    L0, E0, b0 = _problem(N, n, m, 3)
    one = [_dev(a, dtype) for a in (L0, E0, b0)]
    many = [_dev(np.tile(a, (B, 1, 1, 1)), dtype) for a in (L0, E0, b0)]
    for arrays in (one, many):
        create_cholesky_factor_and_solve_launch(*arrays, dtype=dtype)()
    torch.cuda.synchronize()
    for a, b in zip(one, many):
        assert torch.equal(a.expand_as(b), b)


def test_subnormal_pivots():
    """Blocks scaled so that every pivot is subnormal (1e-310 and below) still factor: the fast
    reciprocal square root flushes them, the tile starts over with the library's.  The pivots
    carry 10 bits less than 2^-52 (1e-310 is 2^-1030), so two digits are lost, not more."""
    N, n = 3, 12
    L0 = np.stack([np.diag(np.full(n, 1e-310))] * N)
    E0 = np.zeros((calculate_off_diag_storage_len(N), n, n))
    L, E = _dev(L0, torch.float64), _dev(E0, torch.float64)
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    create_cholesky_factor_launch(L, E, info=info)()
    torch.cuda.synchronize()
    assert info.tolist() == [0]
    diag = torch.diagonal(L, dim1=-2, dim2=-1).cpu().numpy()
    assert np.abs(diag / np.sqrt(1e-310) - 1.0).max() <= 1e-12
