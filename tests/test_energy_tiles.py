"""The pair energies, virial terms and pair gradients of the observables and
of the potential energy on the pair tiles, at the tiles' edges (one particle,
a full tile, one more, several tiles, more entries than a warp's gradient
store holds), against the oracle.  Same tolerance as every FP64 observable:
1e-10 of the value, here of the largest term that enters it.
"""
import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_cases import ANG, MEV, case, momenta, pk, ring, ring_separated

pytestmark = pytest.mark.gpu

KINDS = {
    # pairs inside and outside the damping radius, half-box images
    "aziz_pbc": (dict(T_K=1.5, mass_amu=4.0026, pbc=True, inter="aziz"), 2.0),
    # no cutoff: every pair is an entry, chunked above 384
    "aziz_all": (dict(T_K=1.5, mass_amu=4.0026, inter="aziz"), 2.0),
    "dipole_2d_all": (dict(ndim=2, T_K=2.0, inter="dipole", int_p=(2.4799673e-4, 0, 0)), 1.0),
    "dipole_pbc": (dict(T_K=2.0, pbc=True, inter="dipole", int_p=(2.4799673e-4, 0, 0)), 1.0),
    "harmonic_1d": (dict(ndim=1, T_K=2.0, inter="harmonic", int_p=(1 * MEV, 0, 0), bosonic=False), None),
}


@pytest.mark.parametrize("N", [1, 2, 31, 32, 33, 65, 97])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_observables_and_energy(kind, N):
    kw, dmin = KINDS[kind]
    D = kw.get("ndim", 3)
    box = 3.0 * (N + 8) ** (1.0 / D)
    if kw.get("pbc"):
        kw = dict(kw, cutoff_ang=0.45 * box)
    s, cfg = case(natoms=N, nbeads=3, box_ang=box, **kw)
    x = ring_separated(s, seed=N, dmin_ang=dmin, spread_ang=0.1) if dmin else ring(s, seed=N, spread_ang=0.3)
    p = momenta(s, N)
    want = O.observables(s, x, p)
    with pk.System(cfg) as g:
        g.set_state(x, p)
        got = g.observables()
        terms = g.potential_energy()
        again = g.observables()
    pair = sum(abs(want[k]) for k in ("potential", "int_pot", "virial"))
    for k, v in want.items():
        size = abs(v) + (pair if k in ("potential", "int_pot", "virial") else 0.0)
        assert abs(got[k] - v) <= 1e-10 * size + 1e-300, (k, got[k], v)
    # a second evaluation: the same bits (the exchange's own terms aside, which start from a new estimate)
    assert all(again[k] == got[k] for k in ("potential", "int_pot", "ext_pot", "virial", "w_gsf", "pot_gsf"))
    assert abs(terms[1] - want["int_pot"] * s.nbeads) <= 1e-10 * pair * s.nbeads + 1e-300
    assert abs(terms[0] - want["ext_pot"] * s.nbeads) <= 1e-10 * abs(terms[0])
