"""FP64 charge assignment with charges of very different size in one brick: the
nodes that only small charges reach are as accurate, relative to those charges,
as without the large ones; the result does not depend on the particles' order.

One group of particles per corner of a brick, their stencils disjoint; one or
two CTAs per brick (mesh 64, 32), one or several chunks of particles.

Tolerance: mesh spacing 1, so stencil offsets are exact. A weight (at most 0.55)
rounds at no more than 4 2^-53, a product of three with its charge at 4.5e-16 on
either side: 9e-16 of the group's charge for each of its particles that reach a
node.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

CORNERS = [(x, y, z) for z in (0, 9) for y in (0, 9) for x in (0, 9)]
SIZES = [1.0, 1e6, 1e12, 1e-9, 7.0, 1e-3, 1e30, 3e-200]


def _system(per, sizes, seed):
    rng = np.random.default_rng(seed)
    pos, Z, group = [], [], []
    for g, size in enumerate(sizes):
        pos.append(np.array(CORNERS[g]) + 3.0 * rng.random((per, 3)))
        Z.append(size * rng.choice([1.0, -1.0, 0.75], per))
        group += [g] * per
    return np.concatenate(pos), np.concatenate(Z), np.array(group)


@pytest.mark.parametrize("M", [32, 64])
@pytest.mark.parametrize("per", [1, 20, 70])
@pytest.mark.parametrize("count", [1, 2, 5, 8])
def test_unequal_charges(count, per, M):
    from p3m_b200 import FP64, Context, Replica

    L = float(M)
    pos, Z, group = _system(per, SIZES[:count], 100 * count + per)
    order = np.random.default_rng(1).permutation(len(pos))
    r = Replica(N=len(pos), L=L, kappa=1.0, alpha=1.0, rc=1.0, M=M, skin=0.0)  # short lists
    with Context(r, precision=FP64) as c:
        rho = c.assign(pos, Z)
        shuffled = c.assign(pos[order], Z[order])
    assert np.array_equal(rho, shuffled)
    for g in range(count):
        sel = group == g
        ref = O.assign6(pos[sel], Z[sel], M, M, M, 1.0, 1.0, 1.0)
        x, y, z = CORNERS[g]
        box = (slice(z, z + 9), slice(y, y + 9), slice(x, x + 9))
        assert np.max(np.abs(ref[box])) > 0.0
        err = np.max(np.abs(rho[box] - ref[box]))
        assert err <= per * 9e-16 * SIZES[g], (g, err / SIZES[g])
    assert abs(rho.sum() - Z.sum()) <= 1e-12 * np.abs(Z).sum()
