"""The exchange's weights by rows and by tiles, on both sides of the size where
one takes over from the other, where the weights are banded (a liquid) and
where none is zero (a trap), from a fresh and from a reused estimate.  V and
V_backwards against the oracle, to 1e-10 of the largest potential as
everywhere.
"""
import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_cases import MEV, case, pk, ring

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("liquid", [False, True])
@pytest.mark.parametrize("N", [511, 512, 513, 768, 1023, 1024, 1025])
def test_potentials(N, liquid):
    kw = dict(T_K=1.0, mass_amu=4.0026, pbc=True, box_ang=(N / 0.0218) ** (1 / 3)) if liquid else \
        dict(T_K=2.0, ext="harmonic", ext_p=(3.0 * MEV, 0, 0))
    s, cfg = case(natoms=N, nbeads=3, **kw)
    x = ring(s, seed=N, spread_ang=0.3)
    ref = O.exchange(s, x)
    with pk.System(cfg) as g:
        g.set_state(x, np.zeros_like(x))
        for _ in range(2):
            g.exchange()
            arr = g.exchange_arrays()
            for k in ("V", "Vb"):
                assert np.abs(arr[k] - ref[k]).max() <= 1e-10 * np.abs(ref["V"]).max()
