"""Nose-Hoover chains kept in registers (lengths 2 to 5) and in memory (all
others): trajectories against the oracle's restatement of the reference's
singleChainStep (src/thermostats/nose_hoover.cpp:98-144), for one chain per
bead, per particle and per degree of freedom.

Tolerance: the bound of every trajectory test of these chains, 1e-9 of a
bead's largest element after 12 steps."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_cases import case, momenta, pk, rel_per_bead, ring

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("thermostat", ["nose_hoover", "nose_hoover_np", "nose_hoover_np_dim"])
@pytest.mark.parametrize("nchains", [2, 3, 4, 5, 6])
def test_chain_lengths(thermostat, nchains):
    s, cfg = case(natoms=33, nbeads=4, bosonic=False, thermostat=thermostat, fixcom=False, ext="harmonic",
                  ext_p=(3.0 * 0.036749326e-3, 0, 0), dt_fs=0.5)
    s.nchains = cfg.nchains = nchains
    x = ring(s, seed=29, spread_ang=0.2)
    p = momenta(s, 29)
    tr = O.Trajectory(s, x, p)
    noise = np.zeros((2,) + x.shape)
    with pk.System(cfg) as g:
        g.set_state(x, p)
        for st in range(12):
            assert tr.step(noise) == 0
            g.step(1)
        for got, want in zip(g.get_state(), (tr.x, tr.p, tr.f)):
            assert rel_per_bead(got, want) < 1e-9
        ob = g.observables()
    assert abs(ob["nh_energy"] - tr.nh_energy()) <= 1e-9 * abs(tr.nh_energy())
