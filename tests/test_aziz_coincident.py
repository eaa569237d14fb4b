"""Aziz forces of two particles from nearly coincident (r below 1e-7 of the
potential's length, where the damping is an exponential of minus 1e14) to the
cutoff, in a periodic box, one system and batched.  Against the oracle, with
the tolerance of every FP64 force, 1e-10 of the largest.
"""
import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_cases import case, pk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pbc,cutoff", [(True, 8.0), (False, 8.0), (False, -1.0)])
@pytest.mark.parametrize("r", [5e-7, 2.6e-7, 7.3e-8, 3.8e-8, 2e-8, 5.6e-9, 2.9e-9, 8e-10, 1e-6, 1e-3, 0.5, 3.0, 7.0, 14.0])
def test_two_particles(r, pbc, cutoff):
    s, cfg = case(natoms=2, nbeads=3, mass_amu=4.0026, bosonic=False, pbc=pbc, box_ang=20.0, inter="aziz",
                  cutoff_ang=cutoff)
    x = np.zeros((3, 2, 3))
    x[:, 1, 2] = [r, 1.1 * r, 0.9 * r]
    want = O.update_forces(s, x)["f"]
    with pk.System(cfg) as g, pk.Batch([cfg]) as b:
        g.set_state(x, np.zeros_like(x))
        g.compute_forces()
        b.set_states([x], [np.zeros_like(x)])
        b.compute_forces()
        for f in (g.get_state()[2], b.get_states()[2][0]):
            assert np.abs(f - want).max() <= 1e-10 * np.abs(want).max()
