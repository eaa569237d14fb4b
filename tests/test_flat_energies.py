"""The tile kernels of the cycle energies (from the links' prefix sums) and of
the exchange weights, which large systems use, forced on at the edges of the
tiles and of the prefix blocks; under PBC with pairs at the half-box edge,
where the image must be chosen in FP64.  Against the oracle, to 1e-10 of the
largest value as everywhere (cycle energies of long cycles are sums of up to N
links, each rounded to 2^-53 of the largest).
"""
import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_cases import MEV, case, pk, ring

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ndim", [1, 2, 3])
@pytest.mark.parametrize("pbc", [False, True])
@pytest.mark.parametrize("N", [1, 2, 31, 32, 33, 64, 127, 128, 129, 300])
def test_against_oracle(N, pbc, ndim):
    s, cfg = case(ndim=ndim, natoms=N, nbeads=3, T_K=2.0, ext="harmonic", ext_p=(3.0 * MEV, 0, 0), pbc=pbc,
                  box_ang=8.0)
    x = ring(s, seed=N, spread_ang=0.4)
    if N > 2:  # bead P's particle 0 half a box, and half a box within 1e-9, from bead 1's 1 and 2
        x[0, 1] = x[-1, 0] + 0.5 * s.size
        x[0, 2] = x[-1, 0] + 0.5 * s.size * (1 + 2e-9)
    ref = O.exchange(s, x)
    with pk.System(cfg) as g:
        g.set_option("flat_energies", 1)
        g.set_state(x, np.zeros_like(x))
        got = g.exchange()
        arr = g.exchange_arrays()
    assert np.abs(arr["E"] - ref["E"]).max() <= 1e-10 * ref["E"].max()
    for k in ("V", "Vb"):
        assert np.abs(arr[k] - ref[k]).max() <= 1e-10 * np.abs(ref[k]).max() + 1e-300
    # (exactly half a box apart, the direction of a force is the reference's rounding of dx / L + 1/2)
    for k in ("f1", "fP") if not pbc else ():
        assert np.abs(got[k] - ref[k]).max() <= 1e-10 * np.abs(ref[k]).max()
