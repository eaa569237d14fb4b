"""Exchange potentials of rings stretched far beyond equilibrium, from a fresh
estimate: every link costs up to 1e8 kT, so that the terms of a weight's
exponent, up to 1e11 kT, nearly cancel and no longer fit 32 bits beside it.
V and V_backwards against the oracle.

Tolerance: as at ordinary lengths (test_band_solve), 1e-12 of the largest
potential.
"""
import math

import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_cases import case, pk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kT", [1e0, 1e2, 1e4, 1e5, 1e6, 1e7, 1e8])
@pytest.mark.parametrize("N", [2, 5, 33, 64, 250, 600])
def test_every_link_costs(N, kT):
    s, cfg = case(natoms=N, nbeads=3, T_K=1.0)
    rng = np.random.default_rng(N)
    a = math.sqrt(2 / (s.beta_ex * s.spring_constant))  # a link this long costs 1 kT
    x = rng.normal(0.0, 0.5 * a, (3, N, 3))
    x[-1, :, 0] += a * math.sqrt(kT)
    ref = O.exchange(s, x)
    with pk.System(cfg) as g:
        g.set_state(x, np.zeros_like(x))
        got = g.exchange()
        arr = g.exchange_arrays()
    top = np.abs(ref["V"]).max()
    for k in ("V", "Vb"):
        assert np.abs(arr[k] - ref[k]).max() <= 1e-12 * top, k
    assert abs(got["VB"] - ref["VB"]) <= 1e-12 * top
