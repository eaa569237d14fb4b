"""The exchange estimators (primEstimator and the topology probabilities,
quadratic_bosonic_exchange.cpp:222-279), which the GPU sums over the rows of
the connection probabilities instead of the reference's recursion, against
the oracle's recursion: one row and one chunk, the edges of the 32-entry
chunks and of the eight-row blocks, more rows than the grid has warps, dense
and banded weights, and the exact level-by-level evaluation.

Tolerance: every probability is an exponential of beta_ex times a difference
of potentials and cycle energies, each rounded to 2^-53 of its size, and the
chains of the recursions add up to a few such roundings: 16 units of
beta_ex max(|V|, E) 2^-52, and 1e-12 for the sums.
"""
import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_cases import MEV, case, pk, ring

pytestmark = pytest.mark.gpu

TRAP = dict(T_K=2.0, ext="harmonic", ext_p=(3.0 * MEV, 0, 0))
LIQUID = dict(T_K=1.0, mass_amu=4.0026, pbc=True)


def check(got, s, x):
    ref = O.exchange(s, x)
    size = s.beta_ex * max(np.abs(ref["V"]).max(), ref["E"].max())
    tol = 1e-12 + 16 * 2.0 ** -52 * size
    assert abs(got["prim"] - ref["prim"]) <= tol * abs(ref["prim"])
    for k in ("p_distinct", "p_longest"):
        assert abs(got[k] - ref[k]) <= tol * ref[k] + 1e-300


@pytest.mark.parametrize("N", [1, 2, 8, 9, 31, 32, 33, 65, 257, 2440])
def test_dense_rows(N):
    s, cfg = case(natoms=N, nbeads=3, **TRAP)
    x = ring(s, seed=N, spread_ang=0.5)
    with pk.System(cfg) as g:
        g.set_state(x, np.zeros_like(x))
        check(g.exchange(), s, x)


@pytest.mark.parametrize("N,exact", [(40, 0), (300, 0), (800, 0), (40, 1)])
def test_banded_rows_and_exact_recursion(N, exact):
    s, cfg = case(natoms=N, nbeads=4, box_ang=(N / 0.0218) ** (1 / 3), **LIQUID)
    x = ring(s, seed=N, spread_ang=0.1)
    with pk.System(cfg) as g:
        g.set_option("exact_exchange", exact)
        g.set_state(x, np.zeros_like(x))
        check(g.exchange(), s, x)
