"""The largest system whose pair forces still have room for the tiles' partial
sums (512 MiB of them and the task counters) takes the tiles: two launches, the
tiles and the finishing kernel; one bead more takes the all-pairs kernel, one
launch.  With the same forces.

Tolerance: both are FP64 sums of the same pair forces in different orders,
1e-10 of a bead's largest force as for every FP64 force.
"""
import numpy as np
import pytest

from tests.gpu_cases import case, pk, rel_per_bead

pytestmark = pytest.mark.gpu


def test_the_last_system_on_the_tiles():
    N = 1024
    most = ((512 << 20) // 8 - 1) // (32 * N)  # beads: 32 slots of N doubles each in one dimension
    rng = np.random.default_rng(1)
    x0 = 6.0 * np.arange(N)[:, None] + rng.uniform(-1, 1, (N, 1))
    f = []
    for P, launches in ((most, 2), (most + 1, 1)):
        s, cfg = case(ndim=1, natoms=N, nbeads=P, mass_amu=4.0026, bosonic=False, pbc=True, box_ang=3600.0,
                      inter="aziz", cutoff_ang=1500.0)
        with pk.System(cfg) as g:
            g.set_state(np.repeat(x0[None], P, 0), np.zeros((P, N, 1)))
            before = g.profile(-1)["launches"]
            g.compute_forces()
            assert g.profile(-1)["launches"] - before == launches
            f.append(g.get_state()[2])
    assert rel_per_bead(f[0][:3], f[1][:3]) <= 1e-10
