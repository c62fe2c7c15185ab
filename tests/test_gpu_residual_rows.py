"""GPU: the block-row residual and the refinement set-up over block sizes and right-hand sides.

Tolerances: a sum of 3 n products in any order is within (3 n + 4) eps of the
sum of magnitudes, and the oracle's own sum has the same bound; the backward
error of one refinement round is such a residual over exact norms.
"""
import numpy as np
import pytest
import torch

from oracle import generators, nd_cholesky as nd
from socu_b200.mixed import block_tridiag_residual, create_cholesky_refined_solve_launch

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps
# tile edges, odd sizes (no pair loads), lanes per row (set-up), two column pairs per lane (n > 64)
SIZES = [1, 2, 3, 7, 8, 9, 16, 17, 31, 32, 34, 63, 64, 65, 66, 100, 127, 128]


def _t(a):
    return torch.tensor(a, dtype=torch.float64, device="cuda")


@pytest.mark.parametrize("m", [1, 8, 9, 16, 17, 33])
@pytest.mark.parametrize("n", SIZES)
def test_residual_is_within_rounding(n, m):
    N = 5
    L, E, b = generators.readme_problem(N, n, m, shift=10.0, seed=n)
    x = np.random.default_rng(m).standard_normal(b.shape)
    r = block_tridiag_residual(_t(L), _t(E), _t(x), _t(b)).cpu().numpy()
    ref = b - nd.block_tridiag_matmul(L, E, x)[0]
    scale = np.abs(b) + nd.block_tridiag_matmul(np.abs(L), np.abs(E), np.abs(x))[0]
    assert (np.abs(r - ref) <= 2 * (3 * n + 4) * EPS * scale).all()


@pytest.mark.parametrize("n", SIZES)
def test_backward_error_of_one_round(n):
    N, m = 6, 3
    L, E, b = generators.readme_problem(N, n, m, shift=10.0, seed=n)
    x = torch.zeros(1, N, n, m, dtype=torch.float64, device="cuda")
    run = create_cholesky_refined_solve_launch(_t(L)[None], _t(E)[None], _t(b)[None], x, tol=0.0, max_iter=1,
                                               use_cuda_graph=False)
    run()
    torch.cuda.synchronize()
    ref = nd.backward_error(L, E, x[0].cpu().numpy(), b)[0]
    assert abs(float(run.eta[0]) - ref) <= 2 * (3 * n + 4) * EPS * (1 + 3 * n * ref)
