"""The influence function where its symmetry reduction can go wrong: odd and
even meshes (an even one has a Nyquist component of one sign), small ones, mesh
sides that leave partly filled blocks, and alias ranges and orders around the
eight lanes that share a point.

Tolerance: away from the Nyquist component, whose aliases cancel in pairs,
every sum is dominated by its central term, and both sides add at most 3375
terms in FP64: 1e-12 of the largest value, as for the other influence-function
tests.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,p,m", [(3, 6, 3), (4, 1, 7), (5, 6, 1), (8, 7, 4), (15, 6, 3),
                                   (16, 6, 0), (32, 6, 3), (33, 4, 2), (64, 6, 3)])
def test_gf_opt(M, p, m):
    import yukawa_gf_opt

    kappa, alpha, L = 0.7, 0.33 * M / 20.0, 20.0
    h = L / M
    args = (kappa, alpha, p, m, m, m, M, M, M, h, h, h, L, L, L)
    G, kx, ky, kz, A = yukawa_gf_opt.gf_opt(*args)
    G_ref, kx_ref, ky_ref, kz_ref, A_ref = O.gf_opt(*args)
    assert np.max(np.abs(G - G_ref)) <= 1e-12 * np.max(np.abs(G_ref))
    assert A == pytest.approx(A_ref, rel=1e-12)
    assert np.array_equal(kx, kx_ref) and np.array_equal(ky, ky_ref) and np.array_equal(kz, kz_ref)
