"""FP64 dipole forces of every pair where particle 0, the origin of the
double-float coordinates, lies far outside the cloud of the others, and where
the cloud is two distant groups: separations are then small beside the
coordinates.  Against extended precision, few beads (every pair in FP64) and
many (near pairs in FP64, far ones in double-float).

Tolerance: as for an ordinary cloud (test_dipole_near_far), 2^-48 of the sum
of the pair forces' sizes; the largest coordinate does not enter it.
"""
import numpy as np
import pytest

from tests.test_dipole_near_far import check

pytestmark = pytest.mark.gpu


def cloud(N, ndim, seed):
    rng = np.random.default_rng(seed)
    m = int(np.ceil(N ** (1 / ndim)))
    k = np.arange(N)
    return np.stack([(k // m ** a) % m for a in range(ndim)], 1) * 2.0 + rng.uniform(-0.5, 0.5, (N, ndim))


@pytest.mark.parametrize("nbeads", [1, 640])
@pytest.mark.parametrize("ndim", [2, 3])
@pytest.mark.parametrize("distance", [0.0, 3.0e2, 1.0e4, 1.0e6, 1.0e8])
def test_particle_0_outside(distance, ndim, nbeads):
    x = cloud(130, ndim, 1)
    x[0] += distance
    check(x, ndim, nbeads)


@pytest.mark.parametrize("nbeads", [1, 640])
@pytest.mark.parametrize("distance", [1.0e3, 1.0e6])
def test_two_groups(distance, nbeads):
    x = cloud(130, 2, 2)
    x[65:, 1] -= distance
    check(x, 2, nbeads)
