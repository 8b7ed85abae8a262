"""Calls without a context give large device buffers back before they return, as
a caller with a fixed memory budget needs: what the device has free after a call
is what it had before, but for at most 64 MiB kept for the next call (and the
2 MiB blocks the driver maps memory in)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEPT = (64 + 8) << 20


def _free():
    import torch

    return torch.cuda.mem_get_info()[0]


def test_influence_function():
    from p3m_b200.context import gf_opt_device

    gf_opt_device(1.0, 0.6, 6, 1, 32, 20.0)  # loads the kernels
    before = _free()
    gf_opt_device(1.0, 0.6, 6, 1, 256, 20.0)  # 128 MiB
    assert _free() >= before - KEPT


def test_spectra():
    from p3m_b200.context import sqw_runs

    rng = np.random.default_rng(0)
    a = rng.standard_normal((2, 16384, 3 * 32, 3)) + 0j  # 144 MiB
    sqw_runs(a[:1, :512].copy(), 32, 100.0, 0.1, 51.2)
    before = _free()
    sqw_runs(a, 32, 100.0, 0.1, 1638.4)
    assert _free() >= before - KEPT


def test_error_estimates():
    from p3m_b200.params import pm_error

    pm_error(1000, 16.0, 1.0, 0.6, 32)
    before = _free()
    pm_error(1000, 16.0, 1.0, np.linspace(0.5, 0.7, 200), 256, m_alias=1)
    assert _free() >= before - KEPT
