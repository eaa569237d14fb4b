"""The harmonic interaction of every pair (no cutoff, no images) from the
bead's sum, one system and batched, in FP64: at the edges of the warps and of
the block, with the cloud near the origin and far from it, against extended
precision.

Tolerance: y = x - x_0 is rounded to 2^-53 of itself and enters N times; the
result is rounded to 2^-53 of itself: 2^-52 k N max|y|, twice for the sum over
the particles' roundings.
"""
import numpy as np
import pytest

from tests.gpu_cases import MEV, case, pk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0.0, 1.0e4])
@pytest.mark.parametrize("ndim", [1, 2, 3])
@pytest.mark.parametrize("N", [1, 2, 31, 32, 33, 127, 128, 129, 400])
def test_forces(N, ndim, shift):
    s, cfg = case(ndim=ndim, natoms=N, nbeads=1, inter="harmonic", int_p=(1.0 * MEV, 0, 0), bosonic=False)
    rng = np.random.default_rng(N)
    x = rng.normal(0.0, 5.0, (1, N, ndim)) + shift
    k = s.mass * np.longdouble(1.0 * MEV) ** 2
    xl = x[0].astype(np.longdouble)
    want = -k * (N * xl - xl.sum(0))
    tol = 2.0 ** -51 * float(k) * N * np.abs(x[0] - x[0, 0]).max()
    with pk.System(cfg) as g, pk.Batch([cfg]) as b:
        g.set_state(x, np.zeros_like(x))
        g.compute_forces()
        b.set_states([x], [np.zeros_like(x)])
        b.compute_forces()
        for f in (g.get_state()[2], b.get_states()[2][0]):
            assert np.abs(f[0] - want).max() <= tol
