"""The factorial exchange where links compete for the same targets and even the
cheapest permutation lies thousands of kT above the rows' and columns' minima,
at the sizes whose permutations can no longer be listed: the kernel shifts by
the optimal assignment's potentials.  V_B against the sum over subsets in
logarithms here.

Tolerance: as where the permutations can be listed (test_factorial_subsets).
"""
import math

import numpy as np
import pytest

from tests.gpu_cases import MEV, case, pk

pytestmark = pytest.mark.gpu


def log_permanent(e):
    """log of the sum over permutations of exp(-sum of e)."""
    N = len(e)
    F = np.full(1 << N, -np.inf)
    F[0] = 0.0
    for c in sorted(range(1, 1 << N), key=lambda c: bin(c).count("1")):
        m = [k for k in range(N) if c >> k & 1]
        F[c] = np.logaddexp.reduce(F[[c ^ 1 << k for k in m]] - e[len(m) - 1, m])
    return F[-1]


@pytest.mark.parametrize("pattern", ["two groups", "chain", "spread"])
@pytest.mark.parametrize("N", [2, 9, 10, 11, 12])
def test_competing_links(N, pattern):
    s, cfg = case(natoms=N, nbeads=4, T_K=1.0, ext="harmonic", ext_p=(3.0 * MEV, 0, 0), exchange="factorial")
    unit = math.sqrt(2.0 / (s.beta_ex * s.spring_constant))  # a link this long costs 1 kT
    rng = np.random.default_rng(N)
    x = rng.normal(0.0, 0.5 * unit, (4, N, 3))
    if pattern == "two groups":  # one target too few beside most links
        x[-1, N // 2 + 1:, 0] += 60.0 * unit
        x[0, N // 2:, 0] += 60.0 * unit
    elif pattern == "chain":  # every link one place further than its nearest target
        x[-1, :, 0] += 25.0 * unit * np.arange(N)
        x[0, :, 0] += 25.0 * unit * (np.arange(N) + 1.2)
    else:
        x[-1] += rng.uniform(-1, 1, (N, 3)) * 40.0 * unit
        x[0, :, 1] += 50.0 * unit
    e = s.beta_ex * 0.5 * s.spring_constant * ((x[0][None] - x[-1][:, None]) ** 2).sum(2)
    want = -(log_permanent(e) - math.lgamma(N + 1)) / s.beta_ex
    with pk.System(cfg) as g:
        g.set_state(x, np.zeros_like(x))
        got = g.exchange()["VB"]
    tol = 1e-12 + 16 * 2.0 ** -52 * e.max()
    assert abs(got - want) <= tol * max(abs(want), e.max() / s.beta_ex)
