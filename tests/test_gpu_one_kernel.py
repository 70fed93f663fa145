"""The binary64 step in one kernel, forced where a model of this size would
step on pairs: with and without the cached bond lengths, bit for bit, in rows
of 32 and 128 slots."""
import numpy as np
import pytest

from tests.conftest import cuda_available
from tests.gpu_helpers import lattice, pull_bcs, run_integrator

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(),
                                 reason="needs a CUDA GPU")]


@pytest.mark.parametrize("kind", ["euler", "euler_cromer", "velocity_verlet"])
@pytest.mark.parametrize("horizon,width", [(1.8, 32), (3.015, 128)])
def test_length_cache(monkeypatch, kind, horizon, width):
    import probabilistic_peridynamics_gb300 as pp
    from probabilistic_peridynamics_gb300 import integrators
    monkeypatch.setattr(integrators, "worthwhile", lambda *_: False)
    coords, volume, _, family, nlist, n_neigh = lattice(10, 8, 4, 1.0,
                                                        horizon)
    n = len(coords)
    bc_types, bc_values = pull_bcs(coords, 0)
    assert nlist.shape[1] == width
    s = dict(coords=coords, volume=volume, family=family, nlist=nlist,
             n_neigh=n_neigh, bc_types=bc_types, bc_values=bc_values,
             force_bc_types=np.zeros((n, 3), dtype=np.intc),
             force_bc_values=np.zeros((n, 3)), nnodes=n, max_neigh=width,
             densities=None if kind == "euler" else np.full((n, 3), 50.0),
             k=0.01, s0=0.02)
    dt = 0.5 if kind == "euler" else 1.0
    cls = {"euler": pp.EulerCUDA, "euler_cromer": pp.EulerCromerCUDA,
           "velocity_verlet": pp.VelocityVerletCUDA}[kind]
    steps, outs = 60, []
    for cached in (True, False):
        integ = cls(dt=dt) if kind == "euler" else cls(0.5, dt=dt)
        if not cached:
            make = integ._make_fused_args

            def without(make=make):
                a = make()
                a.bond_length = None
                return a
            integ._make_fused_args = without
        outs.append(run_integrator(integ, s, steps,
                                   3e-3 * np.arange(1, steps + 1)))
        assert integ._pairs is None
        assert bool(integ._fargs.bond_length) == cached
    for a, b in zip(*outs):
        assert np.array_equal(a, b)
    assert np.any((outs[0][6] == -1) & (nlist != -1))  # bonds broke
