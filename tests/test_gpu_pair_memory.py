"""A model whose counted pairs do not fit in memory steps in one kernel: the
same results as on pairs."""
import numpy as np
import pytest

from tests.conftest import cuda_available
from tests.gpu_helpers import breaking_setup, run_integrator

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(),
                                 reason="needs a CUDA GPU")]


def _run(monkeypatch, room):
    import probabilistic_peridynamics_gb300 as pp
    from probabilistic_peridynamics_gb300 import pairs
    monkeypatch.setattr(pairs, "_room", lambda size, device: size < room)
    s = breaking_setup("euler")
    nl = s["nlist"]
    nl[nl > np.arange(nl.shape[0])[:, None]] = -1  # from one end only
    s["n_neigh"] = (nl != -1).sum(1).astype(np.intc)
    integ = pp.EulerCUDA(dt=s["dt"])
    steps = 30
    out = run_integrator(integ, s, steps, 3e-3 * np.arange(1, steps + 1))
    return integ, s, out


def test_falls_back(monkeypatch):
    integ, s, one = _run(monkeypatch, 2 ** 40)
    bonds = int(s["n_neigh"].sum())
    assert integ._pairs.struct.npairs == bonds
    # room for what fits() expects of these bonds, not for their pairs
    room = 4 * s["nlist"].size + 52 * bonds + 1
    assert room < 104 * bonds
    integ, _, two = _run(monkeypatch, room)
    assert integ._pairs is None and integ.bond_length_d is not None
    for a, b in zip(one, two):
        assert np.array_equal(a, b)
