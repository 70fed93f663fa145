"""The pair form against the one-kernel form in rows of 256 and 1,024 slots
that are filled to the last, and nearly so: the same bits on every output."""
import numpy as np
import pytest

from tests.conftest import cuda_available
from tests.gpu_helpers import run_integrator

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(),
                                 reason="needs a CUDA GPU")]


def _setup(width, missing):
    """Points in a ball, each a neighbour of all others: ``width - missing``
    neighbours a row."""
    rng = np.random.default_rng(width)
    n = width - missing + 1
    coords = rng.normal(size=(n, 3))
    nl = np.full((n, width), -1, dtype=np.intc)
    nl[:, :n - 1] = [np.delete(np.arange(n), i) for i in range(n)]
    bc_types = np.zeros((n, 3), dtype=np.intc)
    bc_values = np.zeros((n, 3))
    bc_types[:5, 0], bc_values[:5, 0] = 1, -1.0
    bc_types[-5:, 0], bc_values[-5:, 0] = 1, 1.0
    family = np.full(n, n - 1, dtype=np.intc)
    return dict(coords=coords, volume=rng.uniform(0.5, 1.5, n), family=family,
                nlist=nl, n_neigh=family.copy(), bc_types=bc_types,
                bc_values=bc_values,
                force_bc_types=np.zeros((n, 3), dtype=np.intc),
                force_bc_values=np.zeros((n, 3)),
                densities=np.full((n, 3), 50.0), nnodes=n, max_neigh=width,
                k=1e-4, s0=0.02)


@pytest.mark.parametrize("corrections", [False, True])
@pytest.mark.parametrize("width,missing", [(256, 0), (256, 1), (256, 100),
                                           (1024, 0), (1024, 31)])
def test_same_bits(monkeypatch, width, missing, corrections):
    import probabilistic_peridynamics_gb300 as pp
    from probabilistic_peridynamics_gb300 import integrators
    s = _setup(width, missing)
    if corrections:
        s["stiffness_corrections"] = np.random.default_rng(1).uniform(
            0.5, 1.5, s["nlist"].shape)
    steps, outs = 30, []
    for pairs in (False, True):
        monkeypatch.setattr(integrators, "worthwhile", lambda *_: pairs)
        integ = pp.VelocityVerletCUDA(0.5, dt=1.0)
        outs.append(run_integrator(integ, s, steps,
                                   3e-3 * np.arange(1, steps + 1),
                                   use_run=True))
        assert (integ._pairs is not None) == pairs
    for a, b in zip(*outs):
        assert np.array_equal(a, b)
    assert np.any((outs[0][6] == -1) & (s["nlist"] != -1))  # bonds broke
