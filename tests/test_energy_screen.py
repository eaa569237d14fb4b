"""Pair energies of the observables and of the potential energy where FP32
coordinates cannot tell on which side of the cutoff or of the damping radius a
pair is: a cloud, or one particle of it, far from the origin, and a box of many
cutoffs.  Against the oracle on the same coordinates, with the tolerance of
every FP64 observable, 1e-10.
"""
import numpy as np
import pytest

from oracle import oracle as O
from tests.gpu_cases import ANG, MEV, case, momenta, pk, ring_separated

pytestmark = pytest.mark.gpu

KINDS = {
    "aziz": dict(mass_amu=4.0026, inter="aziz"),
    "aziz_cutoff": dict(mass_amu=4.0026, inter="aziz", cutoff_ang=6.0),
    "harmonic_cutoff": dict(inter="harmonic", int_p=(1.0 * MEV, 0, 0), cutoff_ang=6.0),
    "dipole_2d": dict(ndim=2, inter="dipole", int_p=(2.4799673e-4, 0, 0)),
}


def check(s, cfg, x):
    want = O.potential_energy(s, x)[1]
    p = momenta(s, 1)
    with pk.System(cfg) as g:
        g.set_state(x, p)
        got = g.potential_energy()[1]
        obs = g.observables()["int_pot"] * s.nbeads
    assert abs(got - want) <= 1e-10 * abs(want)
    assert abs(obs - want) <= 1e-10 * abs(want)


@pytest.mark.parametrize("N", [33, 97])
@pytest.mark.parametrize("kind", sorted(KINDS))
@pytest.mark.parametrize("shift,which", [(0.0, "all"), (1e4, "all"), (1e6, "all"), (1e8, "all"), (1e8, "first")])
def test_far_from_the_origin(shift, which, kind, N):
    kw = KINDS[kind]
    s, cfg = case(natoms=N, nbeads=3, bosonic=False, box_ang=4.0 * N ** (1 / kw.get("ndim", 3)), **kw)
    x = ring_separated(s, seed=N, dmin_ang=2.0, spread_ang=0.1)
    if which == "all":
        x += shift
    else:
        x[:, 0] += shift
    check(s, cfg, x)


@pytest.mark.parametrize("kind", ["harmonic_cutoff", "aziz_cutoff"])
def test_box_of_many_cutoffs(kind):
    """Pairs a few 1e-5 of the cutoff inside and outside it, near the box's corner."""
    s, cfg = case(natoms=64, nbeads=2, bosonic=False, pbc=True, box_ang=5.0e4, **KINDS[kind])
    rng = np.random.default_rng(5)
    x = np.empty((2, 64, 3))
    step = 40.0 * ANG * np.arange(32)[:, None]
    x[:, :32] = 0.49 * s.size - step + rng.uniform(-1, 1, (2, 32, 3))
    u = rng.normal(size=(2, 32, 3))
    u /= np.linalg.norm(u, axis=2, keepdims=True)
    x[:, 32:] = x[:, :32] + u * s.cutoff * (1 + rng.uniform(-4e-5, 4e-5, (2, 32, 1)))
    check(s, cfg, x)
