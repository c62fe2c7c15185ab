"""GPU: a sweep on a factor with inverses reads only its triangle.

Row r of the forward sweep of one block depends on rows up to r alone, of the
backward sweep on rows from r on: an infinity in a later (earlier) 8-row tile
of a right-hand side leaves the rows of the other tiles as they are, bit for bit.
"""
import numpy as np
import pytest
import torch

from oracle import generators
from socu_b200.block_tridiag_solver import (
    create_cholesky_backward_substitution_launch,
    create_cholesky_factor_launch,
    create_cholesky_forward_substitution_launch,
)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n", [9, 16, 40, 64])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_other_tiles_are_untouched(dtype, n, bad):
    L0, E0, b0 = generators.readme_problem(1, n, 3, shift=10.0 + 2.0 * np.sqrt(n), seed=n)
    L, E = (torch.tensor(a, dtype=dtype, device="cuda") for a in (L0, E0))
    create_cholesky_factor_launch(L, E, dtype=dtype, keep_inverse=True)()
    last = 8 * ((n - 1) // 8)
    for make, row, keep in ((create_cholesky_forward_substitution_launch, n - 1, slice(0, last)),
                            (create_cholesky_backward_substitution_launch, 0, slice(8, n))):
        x, y = (torch.tensor(b0, dtype=dtype, device="cuda") for _ in range(2))
        y.reshape(n, 3)[row, 1] = bad
        for v in (x, y):
            make(L, E, v, dtype=dtype, factor_has_inverse=True)()
        torch.cuda.synchronize()
        assert torch.isfinite(x).all()
        assert torch.equal(x.reshape(n, 3)[keep], y.reshape(n, 3)[keep])
