"""Autotuner (CPU only): knobs that choose nothing never win, whatever the clock says."""
import pytest
import torch

from socu_b200 import _lib, autotune


@pytest.fixture(autouse=True)
def clean_table():
    _lib.load().socu_tuning_clear()
    yield
    _lib.load().socu_tuning_clear()


@pytest.mark.parametrize("dtype,n", [(torch.float64, 16), (torch.float64, 72), (torch.float32, 64)])
def test_noise_is_not_installed(monkeypatch, dtype, n):
    clock = iter(range(1000, 0, -10))   # every trial looks faster than the one before

    def timer(op, dt, settings, L0, E0, b0, reps, warmup):
        return float(next(clock)), b0

    monkeypatch.setattr(autotune, "_time_op", timer)
    best, _, trials = autotune.tune(n, 1, dtype, horizon=3, device="cpu", save=False)
    dead = [k for k in autotune.KNOBS if k not in autotune.EFFECTIVE]
    assert not any(best[k] for k in dead)
    assert not any(autotune.current_settings(dtype, n, 1)[k] for k in dead)
    assert any(best[k] for k in autotune.EFFECTIVE) == (dtype == torch.float32)
    assert len(trials) > 1
