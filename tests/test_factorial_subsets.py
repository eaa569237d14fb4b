"""The factorial exchange's sum over subsets against the sum over all N!
permutations (numpy, weights relative to the cheapest permutation): every
size whose permutations can be listed, and configurations in which the rows'
and columns' minima leave even the cheapest permutation thousands of kT up
(links that compete for the same target), where the kernel shifts by the
optimal assignment's potentials.

Tolerance: the exponents are beta_ex times link energies, each rounded to
2^-53 of its size: 16 units of the largest exponent times 2^-52, and 1e-12.
"""
import itertools
import math

import numpy as np
import pytest

from tests.gpu_cases import ANG, MEV, case, pk, ring

pytestmark = pytest.mark.gpu


def by_permutations(s, x):
    N, D, P = s.natoms, s.ndim, s.nbeads
    x1, xP = x[0], x[P - 1]

    def image(d):
        return d - s.size * np.floor(d / s.size + 0.5) if s.pbc else d

    d = image(x1[None] - xP[:, None])  # [l][m]
    e = 0.5 * s.spring_constant * (d ** 2).sum(2)
    perms = np.array(list(itertools.permutations(range(N))))
    E = e[np.arange(N), perms].sum(1)
    w = np.exp(-s.beta_ex * (E - E.min()))
    M = np.zeros((N, N))
    for l in range(N):
        np.add.at(M[l], perms[:, l], w)
    M /= w.sum()
    fP = s.spring_constant * ((M[:, :, None] * d).sum(1) + image(x[(P - 2) % P] - xP))
    f1 = s.spring_constant * (-(M[:, :, None] * d).sum(0) + image(x[1 % P] - x1))
    VB = E.min() - math.log(w.sum() / math.factorial(N)) / s.beta_ex
    return dict(VB=VB, prim=-(w @ E) / w.sum() / P, f1=f1, fP=fP, top=s.beta_ex * e.max())


def check(s, cfg, x):
    want = by_permutations(s, x)
    with pk.System(cfg) as g:
        g.set_state(x, np.zeros_like(x))
        got = g.exchange()
        g.compute_forces()
        f = g.get_state()[2]
    tol = 1e-12 + 16 * 2.0 ** -52 * want["top"]
    size = want["top"] / s.beta_ex
    assert abs(got["VB"] - want["VB"]) <= tol * max(abs(want["VB"]), size)
    assert abs(got["prim"] - want["prim"]) <= tol * size * s.natoms
    scale = s.spring_constant * np.abs(x).max() * 2
    for k in ("f1", "fP"):
        assert np.abs(got[k] - want[k]).max() <= tol * scale
    assert np.isfinite(f).all()


@pytest.mark.parametrize("pbc", [False, True])
@pytest.mark.parametrize("N", [1, 2, 3, 4, 5, 7, 8])
def test_every_listable_size(N, pbc):
    s, cfg = case(natoms=N, nbeads=3, T_K=2.0, ext="harmonic", ext_p=(3.0 * MEV, 0, 0), pbc=pbc, box_ang=6.0,
                  exchange="factorial", ndim=1 + N % 3)
    check(s, cfg, ring(s, seed=N, spread_ang=0.5))


@pytest.mark.parametrize("N", [3, 5, 8])
def test_competing_links(N):
    s, cfg = case(natoms=N, nbeads=4, T_K=1.0, ext="harmonic", ext_p=(3.0 * MEV, 0, 0), exchange="factorial")
    rng = np.random.default_rng(N)
    x = rng.normal(0.0, 0.05 * ANG, (s.nbeads, N, 3))
    h = N // 2
    far = math.sqrt(2 * 2000.0 / (s.beta_ex * s.spring_constant))  # a link this long costs 2000 kT
    x[-1, h + 1:, 0] += far  # bead P: h + 1 particles near 0, the others far
    x[0, h:, 0] += far       # bead 1: h near 0
    check(s, cfg, x)
