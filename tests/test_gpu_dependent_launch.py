"""GPU: choices of launch that must not change a bit.

* Kernels that start before their predecessor has ended (programmatic dependent
  launch) against plain stream order, SOCU_PDL=0, in every op, with a mask, with
  tensor-core updates, on narrow levels (the forward pull inside the update's
  launch) and wide ones; several runs each.
* One system, whose sweeps share out right-hand sides over thread blocks,
  against the same system many times over, where they do not.
* Blocks on a pair boundary (whole-tile kernels) against blocks one element off it.
"""
import json
import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from oracle import generators
from socu_b200.block_tridiag_solver import (
    create_cholesky_factor_and_solve_launch,
    create_cholesky_factor_launch,
    create_cholesky_solve_launch,
)

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CASES = [  # (B, N, n, m)
    (1, 200, 10, 1), (1, 129, 32, 9), (1, 700, 64, 8), (1, 60, 72, 17), (1, 40, 128, 33), (9, 33, 17, 3), (40, 64, 24, 2),
]

SCRIPT = r"""
import hashlib, json, sys
import numpy as np, torch
from oracle import generators
from socu_b200.block_tridiag_solver import _launch_with_settings
out = {}
for (B, N, n, m) in json.loads(sys.argv[1]):
    P = [generators.readme_problem(N, n, m, shift=10.0 + 2.0 * n ** 0.5, seed=k) for k in range(B)]
    host = [np.stack([q[i] for q in P]) for i in range(3)]
    for dt in (torch.float32, torch.float64):
        mask = torch.arange(B, device="cuda") % 3 != 1 if B > 1 else None
        for name, settings in [("", {})] + ([("tc", {"update_tensor_cores": 1})] if dt == torch.float32 else []):
            for graph in (False, True):
                L, E, x = (torch.tensor(a, dtype=dt, device="cuda") for a in host)
                start = [a.clone() for a in (L, E, x)]
                fs = _launch_with_settings("factor_and_solve", L, E, x, dt, settings, graph, mask)
                runs = []
                for _ in range(4):
                    for a, a0 in zip((L, E, x), start):
                        a.copy_(a0)
                    fs()
                    y = start[2].clone()
                    _launch_with_settings("solve", L, E, y, dt, {}, graph, mask)()
                    torch.cuda.synchronize()
                    runs.append(hashlib.sha256(b"".join(a.cpu().numpy().tobytes() for a in (L, E, x, y))).hexdigest())
                assert len(set(runs)) == 1
                out[f"{B} {N} {n} {m} {dt} {name} {graph}"] = runs[0]
print(json.dumps(out))
"""


def _run(pdl):
    env = dict(os.environ, SOCU_PDL=pdl, PYTHONPATH=ROOT + os.pathsep + os.environ.get("PYTHONPATH", ""))
    r = subprocess.run([sys.executable, "-c", SCRIPT, json.dumps(CASES)], cwd=ROOT, env=env, capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


def test_dependent_launches_change_no_bit():
    assert _run("1") == _run("0")


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n,m", [(12, 9), (32, 17), (64, 33), (100, 33)])
def test_column_shares_change_no_bit(dtype, n, m):
    N, B = 9, 80
    host = generators.readme_problem(N, n, m, shift=10.0 + 2.0 * np.sqrt(n), seed=n)
    got = []
    for copies in (1, B):
        L, E, x = (torch.tensor(np.tile(a, (copies, 1, 1, 1)), dtype=dtype, device="cuda") for a in host)
        y = x.clone()
        create_cholesky_factor_launch(L, E, dtype=dtype)()
        create_cholesky_solve_launch(L, E, y, dtype=dtype)()
        got.append(y)
    torch.cuda.synchronize()
    assert torch.equal(got[0].expand_as(got[1]), got[1])


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("n", [8, 24, 64, 80, 128])
def test_alignment_changes_no_bit(dtype, n):
    N, m = 11, 5
    host = generators.readme_problem(N, n, m, shift=10.0 + 2.0 * np.sqrt(n), seed=n)
    got = []
    for offset in (0, 1):
        v = []
        for a in host:
            t = torch.empty(a.size + offset, dtype=dtype, device="cuda")[offset:].view(a.shape)
            v.append(t.copy_(torch.as_tensor(a)))
        y = v[2].clone()
        create_cholesky_factor_and_solve_launch(*v, dtype=dtype)()
        create_cholesky_solve_launch(v[0], v[1], y, dtype=dtype)()
        got.append(v + [y])
    torch.cuda.synchronize()
    for a, b in zip(*got):
        assert torch.equal(a, b)
