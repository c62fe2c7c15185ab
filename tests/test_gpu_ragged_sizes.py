"""GPU: every kind of block in the one-warp bodies of a ragged batch.

A large batch of n = 24 systems is solved by single warps; a few systems of
other sizes ride along: whole tiles and partial ones, even sizes (loads by
pairs) and odd ones, one to eight tiles.  Factor, inverse and solution against
the oracle to the tolerances of the small batches (1e-10 relative; refined:
backward error 1e-12); alone, the same systems go to block workers.
"""
import numpy as np
import pytest
import torch

from oracle import generators, nd_cholesky as nd
from socu_b200.ragged import RaggedBatch, create_ragged_factor_and_solve_launch, create_ragged_refined_solve_launch

pytestmark = pytest.mark.gpu
BASE, BASE_N = (256, 24, 1), 190
GROUPS = [[(9, 12, 1), (17, 20, 2), (12, 36, 1), (5, 44, 9), (7, 60, 3)],
          [(9, 13, 1), (6, 37, 2), (4, 57, 1), (5, 64, 9), (11, 56, 4)],
          [(30, 8, 1), (12, 16, 4), (9, 40, 1), (6, 48, 17), (3, 2, 1)]]


def _batch(group, base, refine):
    shapes = group + [BASE] * base
    probs = {s: generators.readme_problem(*s, shift=10.0 + 2.0 * np.sqrt(s[1]), seed=s[1]) for s in set(shapes)}
    N, n, m = (np.array([s[j] for s in shapes]) for j in range(3))
    rb = RaggedBatch(N, n, m, dtype=torch.float64, refine=refine)
    return rb, [probs[s] for s in shapes], rb.pack(*[[probs[s][j] for s in shapes] for j in range(3)])


@pytest.mark.parametrize("base", [0, BASE_N])
@pytest.mark.parametrize("group", GROUPS)
def test_plain(group, base):
    rb, probs, (L, E, x) = _batch(group, base, False)
    create_ragged_factor_and_solve_launch(rb, L, E, x)()
    torch.cuda.synchronize()
    assert rb.error_flag() == 0
    for i in list(range(len(group))) + ([rb.count - 1] if base else []):
        Lo, Eo, xo = (a[0] for a in nd.nd_factor_and_solve(*probs[i]))
        got = rb.L_view(L, i).cpu().numpy()
        inv = np.triu(np.linalg.inv(np.tril(Lo)).transpose(0, 2, 1), 1)
        for a, ref in ((np.tril(got), np.tril(Lo)), (np.triu(got, 1), inv), (rb.E_view(E, i).cpu().numpy(), Eo),
                       (rb.x_view(x, i).cpu().numpy(), xo)):
            assert np.abs(a - ref).max() <= 1e-10 * max(1.0, np.abs(ref).max()), probs[i][0].shape


@pytest.mark.parametrize("base", [0, BASE_N])
@pytest.mark.parametrize("group", GROUPS)
def test_refined(group, base):
    rb, probs, (L, E, b) = _batch(group, base, True)
    x = torch.zeros_like(b)
    run = create_ragged_refined_solve_launch(rb, L, E, b, x, tol=1e-12)
    run()
    torch.cuda.synchronize()
    assert rb.error_flag() == 0 and float(run.eta.max()) <= 1e-12
    for i in range(len(group)):
        L0, E0, b0 = probs[i]
        assert nd.backward_error(L0, E0, rb.x_view(x, i).cpu().numpy(), b0)[0] <= 1e-12
