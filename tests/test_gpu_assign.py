"""Charge assignment and gather at the edges of their work splits: one CTA per
brick or several (few bricks), bricks without particles and with all of them,
several chunks of particles per brick, charges of both signs and of very
different sizes.

Tolerances: a node is a sum of at most N products of three weights. FP64: the
products and the oracle's own sum round at 2^-53 each, N 2^-53 < 3e-13 of the
largest node for N <= 2500; the bar is 1e-12. FP32: weights and offsets round
at 2^-24 each, about ten roundings per product: 1e-6.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

#: (mesh, particles, inside one brick): two CTAs per brick at 32, one beyond
CASES = [(32, 1, False), (32, 60, True), (32, 2500, False), (64, 1, True), (64, 60, True),
         (64, 2500, False), (128, 300, False), (256, 257, False)]


def _system(M, n, cluster):
    rng = np.random.default_rng(1000 * M + n)
    L = 20.0
    pos = rng.random((n, 3)) * (L * 16 / M if cluster else L)
    Z = rng.choice([1.0, -1.0, 1e-3, 3.0], n)
    return L, pos, Z


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("M,n,cluster", CASES)
def test_assign_gather(M, n, cluster, prec):
    from p3m_b200 import FP32, FP64, Context, Replica

    L, pos, Z = _system(M, n, cluster)
    h = L / M
    E = [np.random.default_rng(k).standard_normal((M, M, M)) for k in range(3)]
    rho_ref = O.assign6(pos, Z, M, M, M, h, h, h)
    acc_ref, Ep_ref = O.gather6(pos, Z, M, M, M, h, h, h, *E)
    r = Replica(N=n, L=L, kappa=1.0, alpha=1.0, rc=L / 4, M=M)
    with Context(r, precision=FP64 if prec == "fp64" else FP32) as c:
        rho = c.assign(pos, Z)
        again = c.assign(pos, Z)
        acc, Ep = c.gather(pos, Z, *E)
    assert np.array_equal(rho, again)
    assert np.max(np.abs(rho - rho_ref)) <= (1e-12 if prec == "fp64" else 1e-6) * np.max(np.abs(rho_ref))
    # gather: a field value is a weighted mean of 216 nodes of unit variance
    assert np.max(np.abs(Ep - Ep_ref)) <= (1e-13 if prec == "fp64" else 2e-6)
    assert np.max(np.abs(acc - acc_ref)) <= (1e-12 if prec == "fp64" else 2e-5)
