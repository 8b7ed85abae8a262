"""The influence function at scratch limits of the Ewald parameter: every
reciprocal-space term is a Gaussian exp(-(kappa^2 + k^2) / 4 alpha^2), zero for
alpha -> 0 (also where alpha^2 underflows) and 1 for a large one; the result is
finite and the oracle's."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kappa", [0.0, 0.5])
@pytest.mark.parametrize("alpha", [1e-200, 1e-160, 1e-3, 1e3, 1e150])
def test_gf_opt_limits(alpha, kappa):
    from p3m_b200.context import gf_opt_device

    M, L = 8, 20.0
    h = L / M
    G, A = gf_opt_device(kappa, alpha, 6, 2, M, L)
    with np.errstate(all="ignore"):
        G_ref, _, _, _, A_ref = O.gf_opt(kappa, alpha, 6, 2, 2, 2, M, M, M, h, h, h, L, L, L)
    assert np.all(np.isfinite(G_ref))
    assert np.all(np.isfinite(G)) and np.isfinite(A)
    assert np.max(np.abs(G - G_ref)) <= 1e-12 * np.max(np.abs(G_ref))
    assert A == pytest.approx(A_ref, rel=1e-12)
