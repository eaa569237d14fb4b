"""Replicas run by a cluster of CTAs (few replicas) against the same replicas
run by one CTA each (many), at the replica counts where the cluster's size
changes: forces, exchange scalars and short trajectories.

The two differ only in the order of the centre-of-mass sums: 2^-53 of the
momenta a step, times the few steps' growth, 1e-12 as between the batch and
the one-system path.  In mixed precision such a difference may also move the
rounding of an FP32 term here and there: 1e-7 of the largest value.
"""
import numpy as np
import pytest

from tests.gpu_cases import MEV, case, momenta, pk, ring

pytestmark = pytest.mark.gpu

KINDS = [
    dict(natoms=16, nbeads=32, ext="harmonic", ext_p=(3.0 * MEV, 0, 0)),
    dict(natoms=7, nbeads=5, T_K=2.5, ext="harmonic", ext_p=(3.0 * MEV, 0, 0), inter="harmonic",
         int_p=(1.0 * MEV, 0, 0)),
    dict(natoms=40, nbeads=8, T_K=1.5, mass_amu=4.0026, pbc=True, box_ang=12.0, inter="aziz", cutoff_ang=6.0),
    dict(natoms=33, nbeads=3, bosonic=False, inter="dipole", int_p=(2.4799673e-4, 0, 0), thermostat="none"),
    dict(natoms=12, nbeads=12, propagator="normal_modes", nmthermostat=True, ext="harmonic",
         ext_p=(3.0 * MEV, 0, 0)),
    dict(natoms=1, nbeads=4, fixcom=False, ext="harmonic", ext_p=(3.0 * MEV, 0, 0)),
]


def run(kinds, precision):
    cfgs, xs, ps = [], [], []
    for k in kinds:
        s, cfg = case(**KINDS[k], precision=precision)
        cfg.seed, cfg.replica = 100 + k, k
        cfgs.append(cfg)
        xs.append(ring(s, seed=k, spread_ang=0.3))
        ps.append(momenta(s, k))
    with pk.Batch(cfgs) as b:
        b.set_states(xs, ps)
        b.compute_forces()
        f = b.get_states()[2]
        sc = b.exchange()
        b.set_states(xs, ps)
        b.set_step(0)
        b.step(3)
        return f, sc, b.get_states()


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-7)])
@pytest.mark.parametrize("count", [1, 6, 38, 39, 76, 77, 152, 153])
def test_clusters_match_single_ctas(count, precision, tol):
    want = run([r % len(KINDS) for r in range(312)], precision)  # more than the resident CTAs / 2
    got = run([r % len(KINDS) for r in range(count)], precision)

    def close(u, v):
        assert np.abs(u - v).max() <= tol * max(np.abs(v).max(), 1e-300)

    for r in range(count):
        close(got[0][r], want[0][r])
        close(got[1][r], want[1][r])
        for k in range(3):
            close(got[2][k][r], want[2][k][r])
