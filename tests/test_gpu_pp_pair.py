"""FP64 force and energy of one pair, relative to themselves, from close to the
cutoff down to a hundredth of it: a sparse system whose only neighbours are far
needs the far terms as accurate as the near ones.

Tolerance. The box is a power of two and the displacement a multiple of 2^-20, so
coordinates, differences and r^2 are exact. What rounds: the table (4e-16 of the
term), a Horner recurrence and psi - t psi' (at most six roundings of 2^-53), the
reciprocal root (2^-52, cubed in the force) and four products: 2.4e-15 together;
the bar is 4e-15. (The reference's exp and erfcx terms round at some (10 + 4
(alpha r)^2) 2^-53, 7e-15 at the cutoff.)
"""
import mpmath as mp
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = 16.0
FRACTIONS = [0.01, 0.07, 0.2, 0.4, 0.55, 0.7, 0.8, 0.9, 0.96, 0.99, 0.99999]


def _pair(r, kappa, alpha):
    """(phi, F / r) in 40 digits."""
    with mp.workdps(40):
        k, a = mp.mpf(kappa), mp.mpf(alpha)
        ep = mp.exp(k * r) * mp.erfc(a * r + k / (2 * a))
        em = mp.exp(-k * r) * mp.erfc(a * r - k / (2 * a))
        gauss = mp.exp(-a * a * r * r - k * k / (4 * a * a))
        F = (ep * (1 - k * r) + em * (1 + k * r)) / (2 * r * r) + 2 * a / mp.sqrt(mp.pi) * gauss / r
        return (ep + em) / (2 * r), F / r


@pytest.mark.parametrize("tpi", [1, 8])
@pytest.mark.parametrize("kappa,alpha,rc", [(0.5, 0.72, 5.0), (2.0, 0.72, 4.9), (0.0, 0.75, 4.8),
                                            (3.0, 0.65, 5.1), (1.0, 0.3, 3.3), (6.0, 0.85, 2.975),
                                            (9.0, 0.6, 5.3)])
def test_single_pair(kappa, alpha, rc, tpi):
    from p3m_b200 import FP64, Context, Replica

    rng = np.random.default_rng(3)
    with Context(Replica(N=2, L=L, kappa=kappa, alpha=alpha, rc=rc), precision=FP64) as c:
        c.set_pp_config(tpi)
        for f in FRACTIONS:
            d = rng.standard_normal(3)
            d = np.trunc(d / np.linalg.norm(d) * (f * rc) * 2 ** 20) / 2 ** 20
            r = mp.sqrt(sum(mp.mpf(float(v)) ** 2 for v in d))
            assert r < rc
            phi, fr = _pair(r, kappa, alpha)
            pos = np.array([[8.0, 8.0, 8.0], [8.0, 8.0, 8.0] + d])
            U, acc = c.pp(pos)
            want = np.array([float(-fr * mp.mpf(float(v))) for v in d])
            assert abs(U - float(phi)) <= 4e-15 * float(phi), (f, U / float(phi) - 1)
            assert np.all(np.abs(acc[0] - want) <= 4e-15 * np.abs(want)), (f, acc[0] / want - 1)
            assert np.array_equal(acc[1], -acc[0])
