"""The banded exchange solve (FP32 elimination, FP64 residuals; FP64
substitution where the band or the range of y does not allow it) at the edges
of its 32-node blocks, over temperatures that move the band from a few nodes
through 32 and 64 to dense weights, and after jumps of the coordinates, which
put y far from 1.  V and V_backwards against the oracle.

Tolerance: V = Vh - log(y) / beta with y to a few 2^-52, so the error is the
cycle energies' and the oracle's own rounding, sums of up to N terms of the
largest potential's size: 1e-12 of it.
"""
import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_cases import case, pk, ring

pytestmark = pytest.mark.gpu


def system(N, T):
    return case(natoms=N, nbeads=3, T_K=T, mass_amu=4.0026, pbc=True, box_ang=max(4.0, (N / 0.0218) ** (1 / 3)))


def check(g, s, x):
    ref = O.exchange(s, x)
    g.exchange()
    arr = g.exchange_arrays()
    for k in ("V", "Vb"):
        assert np.abs(arr[k] - ref[k]).max() <= 1e-12 * np.abs(ref["V"]).max() + 1e-300, k


@pytest.mark.parametrize("T", [0.3, 0.6, 1.0, 2.0, 4.0, 8.0, 16.0])
@pytest.mark.parametrize("N", [2, 31, 32, 33, 63, 64, 200, 511, 770, 1025])
def test_bands(N, T):
    s, cfg = system(N, T)
    x = ring(s, seed=N, spread_ang=0.05)
    with pk.System(cfg) as g:
        g.set_state(x, np.zeros_like(x))
        check(g, s, x)
        check(g, s, x)  # from the reused estimate: y is near 1


@pytest.mark.parametrize("N", [40, 300, 800])
def test_estimates_far_off(N):
    """Moves of growing size between evaluations: |log y| from near 0 past
    the range of the FP32 corrections to a retry."""
    s, cfg = system(N, 1.0)
    x = ring(s, seed=N, spread_ang=0.1)
    rng = np.random.default_rng(N)
    with pk.System(cfg) as g:
        for step in (0.0, 0.01, 0.05, 0.1, 0.2, 0.5, 1.0, 0.0):
            x = x + rng.normal(0.0, step, x.shape)
            g.set_state(x, np.zeros_like(x))
            check(g, s, x)
