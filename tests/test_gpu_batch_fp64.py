"""FP64: a replica inside a batch is bit-identical to the same replica alone,
energies included, whatever pair tables its neighbours need: one replica of each
interval count (128, 256, 512) and one whose pair function is too steep for a
table (direct terms). Every lane count; equal lanes on both sides, which fix the
order in which a particle's neighbours are summed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, L = 400, 11.9
#: (kappa, alpha) at rc = L / 4, in an order in which the steepest is not last
PARAMS = [(0.1, 0.46), (40.0, 1.5), (6.0, 0.85), (0.0, 0.9)]


def _run(reps, states, tpi):
    from p3m_b200 import FP64, MODE_NVE, MODE_THERMOSTAT, Context

    with Context(reps, precision=FP64) as c:
        c.set_pp_config(tpi)
        for k, (p, v) in enumerate(states):
            c.set_state(k, p, v)
        c.init_forces()
        first = [c.get_state(k)[2] for k in range(len(reps))]
        u0 = [c.replica_stats(k) for k in range(len(reps))]
        c.run(3, MODE_THERMOSTAT)
        c.run(9, MODE_NVE)
        return first, u0, [c.get_state(k) for k in range(len(reps))], c.energies()


@pytest.mark.parametrize("M", [0, 32])
@pytest.mark.parametrize("tpi", [1, 2, 4, 8])
def test_fp64_replica_equals_alone(tpi, M):
    from p3m_b200 import Replica

    rng = np.random.default_rng(5)
    reps = [Replica(N=N, L=L, kappa=k, alpha=a, rc=L / 4, M=M, dt=0.01, T_desired=0.01)
            for k, a in PARAMS]
    states = [(rng.random((N, 3)) * L, 0.05 * rng.standard_normal((N, 3))) for _ in reps]
    first, u0, end, E = _run(reps, states, tpi)
    for k, r in enumerate(reps):
        f1, u1, e1, E1 = _run([r], [states[k]], tpi)
        assert np.array_equal(first[k], f1[0])
        assert u0[k] == u1[0]
        for a, b in zip(end[k], e1[0]):
            assert np.array_equal(a, b)
        assert np.array_equal(E[:, k], E1[:, 0])
        assert np.all(np.isfinite(E1))
