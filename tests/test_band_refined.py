"""The banded exchange solve by FP32 elimination with FP64 residuals, which
takes bands up to 24 from 64 blocks of 32 nodes on (V has N + 1 nodes, V_back-
wards N: at 2015 particles only V, at 2016 both), around those sizes and at
ragged ones, with a band for each of its column widths 8, 16 and 24 and two
beyond, which the FP64 substitution takes; and after jumps of the coordinates,
which put y out of the range of the FP32 corrections.  V and V_backwards
against the recursion in extended precision over the entries within 90 nodes
(those beyond are below e^-700), on the library's cycle energies.

Tolerance: a weight's exponent is the difference of potentials of up to `top`
kT, rounded to 2^-53 of them, and a node's error passes to the next: 2^-52 N
top kT at most (an elimination that stops a digit early would show).
"""
import numpy as np
import pytest

from tests.gpu_cases import case, pk, ring

pytestmark = pytest.mark.gpu
LD = np.longdouble
NEAR = 90


def recursion(E, beta, N):
    """V, V_backwards, and the band: how far below its node a weight above e^-700 lies."""
    E, beta = E.astype(LD), LD(beta)
    V, Vb, band = np.zeros(N + 1, LD), np.zeros(N + 1, LD), 0

    def log_sum(t):
        m = t.max()
        return m + np.log(np.exp(t - m).sum())

    for p in range(N):
        u0, r = max(0, p + 1 - NEAR), p * (p + 1) // 2
        t = -beta * (E[r + u0:r + p + 1] + V[u0:p + 1])
        V[p + 1] = -(log_sum(t) - np.log(LD(p + 1))) / beta
        band = max(band, p + 1 - u0 - int(np.argmax(t + beta * V[p + 1] > -700)))
    for u in range(N - 1, 0, -1):
        p = np.arange(u, min(N, u + NEAR))
        Vb[u] = -log_sum(-beta * (E[p * (p + 1) // 2 + u] + Vb[p + 1]) - np.log((p + 1).astype(LD))) / beta
    return V, Vb, band


def check(g, s):
    g.exchange()
    arr = g.exchange_arrays()
    N = s.natoms
    V, Vb, band = recursion(arr["E"], s.beta_ex, N)
    tol = 2.0 ** -52 * N * float(np.abs(V).max())
    assert np.abs(arr["V"] - V).max() <= tol
    assert np.abs(arr["Vb"][1:] - Vb[1:]).max() <= tol
    return band


def system(N, T):
    return case(natoms=N, nbeads=3, T_K=T, mass_amu=4.0026, pbc=True, box_ang=(N / 0.0218) ** (1 / 3))


@pytest.mark.parametrize("T,least,most", [(6.0, 1, 8), (2.0, 9, 16), (1.0, 17, 24), (0.7, 25, 32), (0.4, 33, 64)])
@pytest.mark.parametrize("N", [2014, 2015, 2016, 2080])
def test_bands(N, T, least, most):
    s, cfg = system(N, T)
    x = ring(s, seed=N, spread_ang=0.05)
    with pk.System(cfg) as g:
        g.set_state(x, np.zeros_like(x))
        assert least <= check(g, s) <= most
        check(g, s)  # from the reused estimate: y is near 1


@pytest.mark.parametrize("N", [2016, 2100])
def test_estimates_far_off(N):
    """Moves of growing size between evaluations: |log y| from near 0 past the
    range of the FP32 corrections, 46, to a retry, above 200."""
    s, cfg = system(N, 1.0)
    x = ring(s, seed=N, spread_ang=0.1)
    rng = np.random.default_rng(N)
    with pk.System(cfg) as g:
        for move in (0.0, 0.002, 0.01, 0.05, 0.2, 1.0, 0.0):
            x = x + rng.normal(0.0, move, x.shape)
            g.set_state(x, np.zeros_like(x))
            check(g, s)
        assert g.exchange_retries() > 0
