"""Huge, infinite and NaN displacements in every form of the binary64 step
against the oracle, bit for bit: such a bond breaks, and NaN propagates,
whichever form a model takes (the plain kernels, one kernel per step, pairs)
and however wide its rows are.
"""
import numpy as np
import pytest

from tests.conftest import cuda_available
from tests.gpu_helpers import lattice, pull_bcs, run_integrator, run_oracle

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(),
                                 reason="needs a CUDA GPU")]

#: name: (fused, pair list); horizons whose rows have 32 and 128 slots.
ROUTES = {"plain": (False, False), "one_kernel": (True, False),
          "pairs": (True, True)}
HORIZONS = {32: 1.8, 128: 3.015}


@pytest.mark.parametrize("spacing", [0.005, 3.0])
@pytest.mark.parametrize("pull", [1e155, 1e160, 1e300, np.inf, np.nan, 1e-3])
@pytest.mark.parametrize("width", sorted(HORIZONS))
@pytest.mark.parametrize("route", sorted(ROUTES))
def test_bits(monkeypatch, route, width, pull, spacing):
    import probabilistic_peridynamics_gb300 as pp
    from probabilistic_peridynamics_gb300 import integrators
    fused, pairs = ROUTES[route]
    monkeypatch.setattr(integrators, "worthwhile", lambda *_: pairs)
    coords, _, _, family, nlist, n_neigh = lattice(6, 5, 4, spacing,
                                                   HORIZONS[width])
    n = coords.shape[0]
    assert nlist.shape[1] == width
    bc_types, bc_values = pull_bcs(coords, 0)
    setup = dict(coords=coords, volume=np.ones(n), family=family, nlist=nlist,
                 n_neigh=n_neigh, bc_types=bc_types, bc_values=bc_values,
                 force_bc_types=np.zeros((n, 3), dtype=np.intc),
                 force_bc_values=np.zeros((n, 3)), nnodes=n, max_neigh=width,
                 k=0.01, s0=0.02, dt=0.5)
    steps = 4
    mags = np.full(steps, pull)
    integ = pp.EulerCUDA(dt=0.5, fused=fused)
    with np.errstate(all="ignore"):
        ref = run_oracle("euler", setup, steps, mags)
        out = run_integrator(integ, setup, steps, mags)
    assert (integ._pairs is not None) == pairs
    for got, want in zip(out, ref):
        assert np.array_equal(got, want, equal_nan=True)
    if not pull < 1.0:
        assert np.any((out[6] == -1) & (nlist != -1))  # bonds broke
