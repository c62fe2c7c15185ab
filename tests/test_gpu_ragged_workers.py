"""GPU: the two kinds of workers of a ragged batch.

A batch with few nodes is solved by thread blocks, a large one by single warps.
Here the shapes that sit at the edges of the one-warp bodies (one short of, at
and past an 8-row tile, odd tile counts, the largest block, one and two nodes,
more right-hand sides than a tile) are solved both ways: alone, and 64 times
over, which is enough nodes for warp workers.  Every copy must have the same
bits, and one must match the oracle to the tolerances of the small batch
(1e-10 relative; refined: backward error 1e-12).  Kernels over NaN run before
each, so that a result which depends on old shared memory is one too.
"""
import numpy as np
import pytest
import torch

from oracle import generators, nd_cholesky as nd
from socu_b200.block_tridiag_solver import calculate_off_diag_storage_len, create_cholesky_factor_and_solve_launch
from socu_b200.ragged import RaggedBatch, create_ragged_factor_and_solve_launch, create_ragged_refined_solve_launch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 9, 1), (2, 1, 2), (37, 7, 1), (64, 8, 4), (129, 15, 3), (100, 16, 9), (40, 17, 1), (33, 24, 4),
          (65, 32, 1), (20, 39, 2), (50, 48, 4), (7, 57, 1), (21, 64, 17)]
COPIES = 64


def _packed(copies, refine):
    nan = [torch.full((1, k, 64, c), float("nan"), dtype=torch.float64, device="cuda")
           for k, c in ((512, 64), (calculate_off_diag_storage_len(512), 64), (512, 8))]
    create_cholesky_factor_and_solve_launch(*nan, use_cuda_graph=False)()
    probs = [generators.readme_problem(N, n, m, shift=10.0 + 2.0 * np.sqrt(n), seed=11 + k)
             for k, (N, n, m) in enumerate(SHAPES)]
    many = SHAPES * copies
    N, n, m = (np.array([s[j] for s in many]) for j in range(3))
    rb = RaggedBatch(N, n, m, dtype=torch.float64, refine=refine)
    return (rb, probs) + rb.pack(*[[p[j] for p in probs] * copies for j in range(3)])


@pytest.mark.parametrize("copies", [1, COPIES])
def test_workers_match_oracle(copies):
    rb, probs, L, E, x = _packed(copies, False)
    create_ragged_factor_and_solve_launch(rb, L, E, x)()
    torch.cuda.synchronize()
    assert rb.error_flag() == 0
    k = len(SHAPES)
    for i, (L0, E0, b0) in enumerate(probs):
        Lo, Eo, xo = (a[0] for a in nd.nd_factor_and_solve(L0, E0, b0))
        for got, ref in ((torch.tril(rb.L_view(L, i)), np.tril(Lo)), (rb.E_view(E, i), Eo), (rb.x_view(x, i), xo)):
            if ref.size:
                assert np.abs(got.cpu().numpy() - ref).max() <= 1e-10 * max(1.0, np.abs(ref).max()), SHAPES[i]
        inv = np.triu(np.linalg.inv(np.tril(Lo)).transpose(0, 2, 1), 1)
        assert np.abs(np.triu(rb.L_view(L, i).cpu().numpy(), 1) - inv).max() <= 1e-10, SHAPES[i]
        for c in range(1, copies):
            assert torch.equal(rb.x_view(x, i), rb.x_view(x, i + c * k)) and torch.equal(
                rb.E_view(E, i), rb.E_view(E, i + c * k)), SHAPES[i]


@pytest.mark.parametrize("copies", [1, COPIES])
def test_refined_workers(copies):
    rb, probs, L, E, b = _packed(copies, True)
    x = torch.zeros_like(b)
    run = create_ragged_refined_solve_launch(rb, L, E, b, x, tol=1e-12)
    run()
    torch.cuda.synchronize()
    assert rb.error_flag() == 0 and float(run.eta.max()) <= 1e-12
    for i, (L0, E0, b0) in enumerate(probs):
        assert nd.backward_error(L0, E0, rb.x_view(x, i).cpu().numpy(), b0)[0] <= 1e-12, SHAPES[i]
