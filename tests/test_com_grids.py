"""Centre-of-mass removal by kernels of different grids on one handle:
zero_momentum (one block per 256 or 1024 pairs) between steps of the Cartesian
propagator with the normal-mode thermostat (one block per four particles and
axis), with neither, either and both grids above the size from which the last
block leaves the mean.  Against a second handle on which the mean is removed
here, in numpy, instead.

Tolerance: the two differ in the rounding of the mean, a few 2^-53 of the
momenta, carried through two steps: 1e-12 of the largest.
"""
import numpy as np
import pytest

from tests.gpu_cases import MEV, case, momenta, pk, ring

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,P", [(40, 8), (700, 20), (400, 300), (1024, 100), (1024, 160), (4096, 32)])
def test_zero_momentum_between_steps(N, P):
    s, cfg = case(natoms=N, nbeads=P, T_K=5.0, bosonic=False, nmthermostat=True, ext="harmonic",
                  ext_p=(3.0 * MEV, 0, 0))
    x, p = ring(s, seed=N), momenta(s, P) + 0.5
    tol = 1e-12 * np.abs(p).max()

    def removed(q):
        return q - q.mean((0, 1))

    with pk.System(cfg) as a, pk.System(cfg) as b:
        a.set_state(x, p)
        b.set_state(x, p)
        for nsteps in (2, 1, 3):
            before = a.get_state()[1]
            a.zero_momentum()
            after = a.get_state()[1]
            assert np.abs(after - removed(before)).max() <= tol
            pb = b.get_state()[1]
            b.set_state(None, removed(pb))
            for g in (a, b):
                g.compute_forces()  # set_state sets them to zero
                g.step(nsteps)
            (xa, pa, _), (xb, pb, _) = a.get_state(), b.get_state()
            assert np.abs(pa - pb).max() <= tol
            assert np.abs(pa.mean((0, 1))).max() <= tol
            assert np.abs(xa - xb).max() <= 1e-12 * np.abs(x).max()
