"""The FP64 harmonic interaction of every pair where particle 0, the origin of
the bead's sum, lies far outside the cloud: one system, at the sizes where the
block's threads take one particle, some two, and many.

Tolerance: the force k (S - N y) with S and y as good as exact takes four
roundings of 2^-53 of itself: 2^-50.
"""
import numpy as np
import pytest

from tests.gpu_cases import MEV, case, pk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("distance", [0.0, 1e1, 1e3, 1e6, 1e9])
@pytest.mark.parametrize("N", [2, 16, 128, 129, 300, 1000])
def test_particle_0_outside(N, distance):
    s, cfg = case(natoms=N, nbeads=3, inter="harmonic", int_p=(1 * MEV, 0, 0), bosonic=False)
    rng = np.random.default_rng(N)
    x = rng.normal(0.0, 5.0, (N, 3))
    x[0] += distance * (1 + rng.uniform(0, 1, 3))
    xl = x.astype(np.longdouble)
    want = np.longdouble(s.mass) * np.longdouble(MEV) ** 2 * (xl.sum(0) - N * xl)
    with pk.System(cfg) as g:
        g.set_state(np.repeat(x[None], 3, 0), np.zeros((3, N, 3)))  # equal beads: no spring forces
        g.compute_forces()
        f = g.get_state()[2]
    assert (f == f[0]).all()
    assert (np.abs(f[0] - want).max(1) <= 2.0 ** -50 * np.abs(want).max(1)).all()
