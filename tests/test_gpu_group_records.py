"""What a captured group of steps records: the n(q,t) rows belong to the steps
they are filed under (inside a group the row index is advanced by the previous
step's reduction, beside the next step), equal to the rows of a run step by step
bit for bit and to the oracle's at that step's positions; and the thermostat's
change of rule after step 1999, inside a group.

Tolerances: an n(q,t) value sums 300 unit phases whose arguments (up to 8 pi)
round at 2^-53 of themselves: 300 x 25 x 1.2e-16 < 1e-12; the bar is 1e-11. The
thermostat's factor is a quotient and a root of recorded numbers: 1e-14.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

N, NQ = 300, 4


def _replica(n, M):
    from p3m_b200 import Replica

    L = (4 * np.pi * n / 3) ** (1 / 3)
    return Replica(N=n, L=L, kappa=2.0, alpha=0.6, rc=L / 3.2, M=M, dt=0.05, T_desired=0.01)


def _context(reps, prec):
    """Particles near the sites of an 8^3 lattice."""
    from p3m_b200 import Context

    rng = np.random.default_rng(23)
    site = np.stack(np.meshgrid(*[np.arange(8)] * 3), -1).reshape(-1, 3)
    c = Context(reps, precision=prec)
    for k, r in enumerate(reps):
        pos = (rng.permutation(site)[:r.N] + 0.5 + 0.1 * rng.standard_normal((r.N, 3))) * (r.L / 8)
        c.set_green(replica=k)
        c.set_state(k, pos % r.L, 0.1 * rng.standard_normal((r.N, 3)))
    c.init_forces()
    c.set_nqt(np.arange(1.0, NQ + 1), 64)
    return c


@pytest.mark.parametrize("prec_name", ["fp32", "fp64"])
@pytest.mark.parametrize("mode_name", ["nve", "thermostat"])
@pytest.mark.parametrize("steps", [9, 17])
def test_nqt_rows(steps, mode_name, prec_name):
    from p3m_b200 import FP32, FP64, MODE_NVE, MODE_THERMOSTAT

    mode = MODE_NVE if mode_name == "nve" else MODE_THERMOSTAT
    prec = FP32 if prec_name == "fp32" else FP64
    reps = [_replica(N, 32), _replica(N + 57, 64)]
    with _context(reps, prec) as c:
        c.run(steps, mode, record_nqt=True)
        rows = [c.get_nqt(k, NQ) for k in range(2)]
    with _context(reps, prec) as c:
        for s in range(steps):
            c.run(1, mode, it0=s, record_nqt=True, graph=False)
            if s in (3, 7, 8, steps - 1):
                for k, r in enumerate(reps):
                    q = 2 * np.pi / r.L * np.arange(1, NQ + 1)
                    ref = O.nqt(c.get_state(k)[0], q)
                    bar = 1e-11 if prec == FP64 else 1e-3  # FP32 phases: 300 x 25 x 6e-8
                    assert np.max(np.abs(rows[k][s] - ref)) <= bar
        for k in range(2):
            assert np.array_equal(rows[k], c.get_nqt(k, NQ))


@pytest.mark.parametrize("prec_name", ["fp32", "fp64"])
@pytest.mark.parametrize("it0,steps", [(1996, 8), (1990, 17), (1999, 9), (2000, 9)])
def test_thermostat_rule_in_a_group(it0, steps, prec_name):
    from p3m_b200 import FP32, FP64, MODE_THERMOSTAT

    prec = FP32 if prec_name == "fp32" else FP64
    reps = [_replica(N, 32), _replica(N + 57, 64)]
    got = []
    for graph in (True, False):
        with _context(reps, prec) as c:
            c.run(12, MODE_THERMOSTAT)
            c.run(steps, MODE_THERMOSTAT, it0=it0, graph=graph)
            got.append((c.energies()[12:], [c.get_state(k) for k in range(2)]))
    assert np.array_equal(got[0][0], got[1][0])
    for a, b in zip(got[0][1], got[1][1]):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
    T, fact = got[0][0][..., 2], got[0][0][..., 3]
    it = (it0 + np.arange(steps))[:, None]
    Td = 0.01
    want = np.where(it <= 1999, np.sqrt(Td / T), np.sqrt((20 * Td / T - 1) / 20))
    assert np.all(np.abs(fact - want) <= 1e-14 * want)
