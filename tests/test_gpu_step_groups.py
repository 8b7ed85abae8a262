"""Several steps captured as one graph leave work to one another (the
thermostat's rescale to the next step's drift, the energy sums beside it, the
brick counts to the last block that reads them): states, energies and the
records of a run in groups are those of the run step by step, bit for bit. Step
counts around the group size of eight; replicas of different meshes, one too
large for the placing pass to sum its brick counts itself."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _replicas(shapes):
    from p3m_b200 import Replica

    out = []
    for n, M in shapes:
        L = (4 * np.pi * n / 3) ** (1 / 3)
        out.append(Replica(N=n, L=L, kappa=2.0, alpha=0.6, rc=L / 3.2, M=M, dt=0.05, T_desired=0.01))
    return out


@pytest.mark.parametrize("prec_name", ["fp32", "fp64"])
@pytest.mark.parametrize("mode_name", ["thermostat", "nve"])
@pytest.mark.parametrize("shapes,steps", [([(300, 32)], 7), ([(513, 64), (200, 32)], 17),
                                          ([(700, 32), (256, 256)], 9)])
def test_groups_equal_single_steps(shapes, steps, mode_name, prec_name):
    from p3m_b200 import FP32, FP64, MODE_NVE, MODE_THERMOSTAT, Context

    reps = _replicas(shapes)
    rng = np.random.default_rng(17)
    pos = [rng.random((r.N, 3)) * r.L for r in reps]
    vel = [0.1 * rng.standard_normal((r.N, 3)) for r in reps]
    mode = MODE_THERMOSTAT if mode_name == "thermostat" else MODE_NVE
    got = []
    for graph in (False, True):
        with Context(reps, precision=FP32 if prec_name == "fp32" else FP64) as c:
            for k in range(len(reps)):
                c.set_green(replica=k)
                c.set_state(k, pos[k], vel[k])
            c.init_forces()
            c.run(steps, mode, graph=graph)
            c.run(steps, MODE_NVE, graph=graph)
            got.append(([c.get_state(k) for k in range(len(reps))], c.energies()))
    for a, b in zip(*[g[0] for g in got]):
        for x, y in zip(a, b):
            assert np.array_equal(x, y)
    assert got[0][1].shape == (2 * steps, len(reps), 4)
    assert np.array_equal(got[0][1], got[1][1])
    assert np.all(np.isfinite(got[0][1]))
