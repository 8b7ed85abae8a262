"""The influence function's error against extended precision, over the whole
(root of summed squares): a few lowest wave vectors carry it, so a factor common
to all of them counts in full.

Tolerance: per value some twenty roundings of 2^-53 to 2^-52 (four exponentials
and their products, three powers of sin x / x, the sums over aliases, dominated by
one term, and a quotient): 5e-16 as independent errors; the bar is 1e-15. (With
the rounding of the exponents, up to (kappa / 2 alpha)^2, and of sin x / x to the
twelfth power it was 0.7 to 3e-15.)
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _exact(points, kappa, alpha, M, L, p, m):
    pi = LD("3.14159265358979323846264338327950288")
    ka, al, L = LD(kappa), LD(alpha), LD(L)
    a = np.arange(-m, m + 1)
    out = []
    for s in points:
        k = 2 * pi * s.astype(LD) / L
        km = 2 * pi * (s[:, None] + a[None] * M).astype(LD) / L
        x = km * (L / M) / 2
        U = np.where(x == 0, LD(1), np.sin(x) / np.where(x == 0, LD(1), x)) ** (2 * p)
        outer = lambda v, op: op(op(v[0][:, None, None], v[1][None, :, None]), v[2][None, None, :])  # noqa: E731
        u, q, dot = outer(U, np.multiply), outer(km ** 2, np.add) + ka ** 2, outer(k[:, None] * km, np.add)
        num = (u * dot * (4 * pi * np.exp(-q / (4 * al ** 2)) / q)).sum()
        out.append(num / (u.sum() ** 2 * (k ** 2).sum()))
    return np.array(out, dtype=LD)


@pytest.mark.parametrize("M", [32, 64, 96, 128])
@pytest.mark.parametrize("n,kappa", [(3000, 0.4), (3000, 2.6), (20000, 0.7), (20000, 1.9), (150000, 3.0)])
def test_error_of_the_whole(n, kappa, M):
    from p3m_b200.context import gf_opt_device

    L = (4 * np.pi * n / 3) ** (1 / 3)
    alpha = 0.331 * M / L
    rng = np.random.default_rng(n + M)
    low = np.stack(np.meshgrid(*[np.arange(-2, 3)] * 3), -1).reshape(-1, 3)
    s = np.concatenate([low[np.any(low != 0, axis=1)], rng.integers(-M // 2 + 1, M // 2, (200, 3))])
    s = s[np.any(s != 0, axis=1)]
    G, _ = gf_opt_device(kappa, alpha, 6, 3, M, L)
    got = G[tuple((s + M // 2)[:, d] for d in range(3))].astype(LD)
    ref = _exact(s, kappa, alpha, M, L, 6, 3)
    err = float(np.sqrt(((got - ref) ** 2).sum() / (ref ** 2).sum()))
    assert err <= 1e-15, err
