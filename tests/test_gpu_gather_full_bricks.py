"""The gather where one brick holds more particles than a CTA has threads (256),
with a CTA per brick and component (up to 512 bricks) as well as a CTA per
brick: each staged tile serves several chunks of particles.

Tolerances as for any gather against the oracle: a field value is a mean of 216
nodes of unit variance with weights of at most ten roundings each: FP64 1e-13,
FP32 2e-6; the acceleration has the factor Z <= 3.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("M,n", [(32, 300), (64, 260), (64, 516), (64, 771), (256, 771)])
def test_full_brick(M, n, mode, prec):
    from p3m_b200 import FP32, FP64, Context, Replica

    rng = np.random.default_rng(M + n)
    L = 20.0
    h = L / M
    pos = rng.random((n, 3)) * (L * 16 / M)
    pos[-3:] = rng.random((3, 3)) * L
    brick = np.floor(pos / (16 * h)).astype(int)
    assert np.unique(brick, axis=0, return_counts=True)[1].max() > 256
    Z = rng.choice([1.0, -1.0, 3.0], n)
    E = [rng.standard_normal((M, M, M)) for _ in range(3)]
    acc_ref, Ep_ref = O.gather6(pos, Z, M, M, M, h, h, h, *E)
    r = Replica(N=n, L=L, kappa=1.0, alpha=1.0, rc=0.25, M=M, skin=0.0)  # short lists
    with Context(r, precision=FP64 if prec == "fp64" else FP32) as c:
        c.set_tuning(gather_mode=mode)
        acc, Ep = c.gather(pos, Z, *E)
    tol = 1e-13 if prec == "fp64" else 2e-6
    assert np.max(np.abs(Ep - Ep_ref)) <= tol
    assert np.max(np.abs(acc - acc_ref)) <= 10 * tol
