"""FP64 pair forces from the table: parameters that take each interval count,
and a pair function too steep for it (direct evaluation); a pair just inside
the cutoff; every lane count.

Tolerance: the table holds psi and g = F r^2 to 4e-16 of psi(0) = 1, so a
pair's force to about 1e-15 of 1/r^2, like the oracle's own arithmetic; the
coordinates round at L 2^-53, 1e-14 of the closest distances of random
positions. Sums of at most a few hundred pairs keep that within 1e-12
(relative RMS), the bar of the direct evaluation.
"""
import numpy as np
import pytest

from gpu_util import rel_rms
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tpi", [1, 2, 4, 8])
@pytest.mark.parametrize("kappa,alpha", [(0.0, 0.9), (0.1, 0.46), (1.0, 0.6), (3.0, 0.45), (6.0, 0.85),
                                         (40.0, 1.5)])
def test_pp_fp64(kappa, alpha, tpi):
    from p3m_b200 import FP64, Context, Replica

    N, L = 400, 11.9
    rc = L / 4
    rng = np.random.default_rng(int(100 * kappa + 10 * alpha))
    pos = rng.random((N, 3)) * L
    pos[3] = (pos[2] + [0.0, rc * (1 - 1e-9), 0.0]) % L
    U_ref, acc_ref = O.pp(kappa, alpha, rc, np.full(3, L), pos)
    with Context(Replica(N=N, L=L, kappa=kappa, alpha=alpha, rc=rc), precision=FP64) as c:
        c.set_pp_config(tpi)
        U, acc = c.pp(pos)
    assert U == pytest.approx(U_ref, rel=1e-12)
    assert rel_rms(acc, acc_ref) < 1e-12
