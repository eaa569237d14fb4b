"""The exchange's fresh FP32 estimate: one block's two halves below 512
particles, CTAs that hand 32-node blocks to one another from there on, at the
edges of the blocks and of the CTAs' round-robin, dense and banded weights;
and the jump of a running system to new coordinates, after which the solve
must go back to a fresh estimate once.

The estimate only has to be near V: the solve corrects it exactly.  So V,
V_backwards and V_B are compared with the oracle's recursion, to 1e-10 of the
largest potential as everywhere; an estimate that is off by more than 200 kT
would be counted as a retry.
"""
import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_cases import MEV, case, momenta, pk, ring

pytestmark = pytest.mark.gpu

TRAP = dict(T_K=2.0, ext="harmonic", ext_p=(3.0 * MEV, 0, 0))


def check(g, s, x):
    ref = O.exchange(s, x)
    got = g.exchange()
    arr = g.exchange_arrays()
    size = np.abs(ref["V"]).max()
    assert abs(got["VB"] - ref["VB"]) <= 1e-10 * size
    assert np.abs(arr["V"] - ref["V"]).max() <= 1e-10 * size
    assert np.abs(arr["Vb"] - ref["Vb"]).max() <= 1e-10 * np.abs(ref["Vb"]).max() + 1e-300


@pytest.mark.parametrize("liquid", [False, True])
@pytest.mark.parametrize("N", [1, 2, 31, 32, 33, 64, 95, 255, 511, 512, 543, 544, 2047, 2080])
def test_fresh_estimate(N, liquid):
    kw = dict(T_K=1.0, mass_amu=4.0026, pbc=True, box_ang=(N / 0.0218) ** (1 / 3)) if liquid else TRAP
    s, cfg = case(natoms=N, nbeads=3, **kw)
    x = ring(s, seed=N, spread_ang=0.4)
    with pk.System(cfg) as g:
        g.set_state(x, np.zeros_like(x))
        check(g, s, x)
        assert g.exchange_fresh_estimates() == 1 and g.exchange_retries() == 0


@pytest.mark.parametrize("N", [40, 300, 900])
def test_jump_to_new_coordinates(N):
    s, cfg = case(natoms=N, nbeads=3, **TRAP)
    xs = [ring(s, seed=k, spread_ang=0.4) for k in (1, 2)]
    p = momenta(s, 1)
    with pk.System(cfg) as g:
        for x in (xs[0], xs[1], xs[0]):
            g.set_state(x, p)
            g.step(3)
            g.set_state(x, p)
            check(g, s, x)
