"""The Aziz pair energy of the observables and of the potential energy over
every distance a pair can have, from nearly coincident particles (r below 1e-7
of the potential's length, where the damping is an exponential of minus 1e14)
to ones thrown far apart.  Against the oracle, with the tolerance of every
FP64 observable, 1e-10.
"""
import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_cases import case, momenta, pk

pytestmark = pytest.mark.gpu

APART = [5e-7, 2e-7, 7.3e-8, 2e-8, 2.9e-9, 1e-3, 0.5, 3.0, 6.9, 7.1, 50.0, 1e4, 3e6, 1e8, 1e11, 4.7e12, 9e12, 1.7e13,
         2.2e14, 1.5e15]


@pytest.mark.parametrize("r", APART)
def test_two_particles(r):
    s, cfg = case(natoms=2, nbeads=2, mass_amu=4.0026, bosonic=False, inter="aziz")
    x = np.zeros((2, 2, 3))
    x[:, 1, 1] = [r, 1.25 * r]
    want = O.potential_energy(s, x)[1]
    with pk.System(cfg) as g:
        g.set_state(x, momenta(s, 1))
        got = g.potential_energy()[1]
        obs = g.observables()["int_pot"] * s.nbeads
    assert abs(got - want) <= 1e-10 * abs(want)
    assert abs(obs - want) <= 1e-10 * abs(want)
