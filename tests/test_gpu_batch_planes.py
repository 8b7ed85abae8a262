"""FP32: a replica in a batch whose y/z FFT planes outnumber the SMs (the plane
kernel then runs with half the threads) is bit-identical to the same replica
alone, field energy and states included; meshes of 64 and 32 points a side, and
a batch of either side of the line (148 planes)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(reps, states):
    from p3m_b200 import FP32, MODE_NVE, Context

    with Context(reps, precision=FP32) as c:
        c.set_pp_config(2)
        for k, (p, v) in enumerate(states):
            c.set_state(k, p, v)
        c.init_forces()
        u = [c.replica_stats(k) for k in range(len(reps))]
        first = [c.get_state(k)[2] for k in range(len(reps))]
        c.run(9, MODE_NVE)
        return u, first, [c.get_state(k) for k in range(len(reps))], c.energies()


@pytest.mark.parametrize("meshes", [[64] * 4 + [32] * 2, [32] * 9, [64] * 4])
def test_batch_of_many_planes_equals_alone(meshes):
    from p3m_b200 import Replica

    rng = np.random.default_rng(len(meshes))
    reps, states = [], []
    for k, M in enumerate(meshes):
        n = 400 + 60 * k
        box = (4 * np.pi * n / 3) ** (1 / 3)
        reps.append(Replica(N=n, L=box, kappa=0.5 + 0.2 * k, alpha=0.8, rc=box / 3.2, M=M, dt=0.02,
                            T_desired=0.01))
        states.append((rng.random((n, 3)) * box, 0.1 * rng.standard_normal((n, 3))))
    u, first, end, E = _run(reps, states)
    for k, r in enumerate(reps):
        u1, f1, e1, E1 = _run([r], [states[k]])
        assert np.array_equal(first[k], f1[0])
        assert u[k] == u1[0]
        for a, b in zip(end[k], e1[0]):
            assert np.array_equal(a, b)
        assert np.array_equal(E[:, k], E1[:, 0])
