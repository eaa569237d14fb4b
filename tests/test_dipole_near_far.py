"""FP64 dipole forces of every pair: near pairs in FP64, far ones in
double-float, at the edges of the tiles, with more near pairs than a warp
holds at once, with a dense cluster beside distant particles, far from the
origin, and at scales where double-floats have no room for r^-5 (all pairs
FP64 then).  Against extended precision.

Tolerance: a pair's FP64 force carries at most about 12 roundings of 2^-53
(the separation, squared twice and a half, the power and the product), a far
pair's 2^-42 of a force that is at most 2^-10 of the nearest one: 2^-48 of the
sum of the pair forces' sizes.  (Double-floats throughout would leave 2^-44.)
"""
import numpy as np
import pytest

from tests.gpu_cases import case, pk

pytestmark = pytest.mark.gpu


def forces(x, ndim, nbeads):
    """Of a bead; all beads at x, so that the springs are zero (few beads: too
    few tiles for the near/far kernels, every pair in FP64)."""
    N = x.shape[0]
    s, cfg = case(ndim=ndim, natoms=N, nbeads=nbeads, inter="dipole", int_p=(2.4799673e-4, 0, 0), bosonic=False)
    with pk.System(cfg) as g:
        g.set_state(np.repeat(x[None], nbeads, 0), np.zeros((nbeads, N, ndim)))
        g.compute_forces()
        f = g.get_state()[2]
    assert (f == f[0]).all()
    return f[0]


def check(x, ndim, nbeads):
    N = x.shape[0]
    f = forces(x, ndim, nbeads)
    xl = x.astype(np.longdouble)
    d = xl[:, None] - xl[None]
    r2 = (d ** 2).sum(2)
    np.fill_diagonal(r2, 1)
    pair = 3 * np.longdouble(2.4799673e-4) * r2 ** np.longdouble(-2.5)
    np.fill_diagonal(pair, 0)
    want = (pair[:, :, None] * d).sum(1)
    size = (pair * np.sqrt(r2)).sum(1)
    assert (np.abs(f - want).max(1) <= 2.0 ** -48 * size).all()


@pytest.mark.parametrize("nbeads", [1, 640])
@pytest.mark.parametrize("ndim", [1, 2, 3])
@pytest.mark.parametrize("N", [1, 2, 31, 32, 33, 65, 200])
def test_scattered(N, ndim, nbeads):
    rng = np.random.default_rng(N)
    if ndim == 1:
        x = (3.0 * np.arange(N) + rng.uniform(-1, 1, N))[:, None]
    else:
        m = int(np.ceil(N ** (1 / ndim)))
        k = np.arange(N)
        x = np.stack([(k // m ** a) % m for a in range(ndim)], 1) * 3.5 + rng.uniform(-1, 1, (N, ndim))
    check(x, ndim, nbeads)


@pytest.mark.parametrize("nbeads", [1, 640])
@pytest.mark.parametrize("scale,shift", [(1.0, 1.0e4), (1.0e-5, 0.0), (1.0e5, 0.0), (1.0e-2, 0.0)])
def test_scales_and_cluster(scale, shift, nbeads):
    rng = np.random.default_rng(3)
    x = rng.uniform(-60, 60, (150, 2))
    x[:70] = rng.uniform(-3, 3, (70, 2))  # a cluster: every pair of its tiles is near
    check(x * scale + shift, 2, nbeads)
