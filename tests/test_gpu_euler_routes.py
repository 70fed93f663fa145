"""Every route of the GPU ``Euler`` against one kernel per Cython function:
the pair form and ``pp_cy_break_and_force``, which takes over where a pair list
does not fit.  Bit-identical on every output, also when the time step and the
material change between two steps.
"""
import numpy as np
import pytest

from tests.conftest import cuda_available
from tests.cython_setup import breaking_lattice
from tests.test_gpu_euler_pairs import _setup

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(),
                                 reason="needs a CUDA GPU")]


def _run(monkeypatch, setup, route, steps, change):
    import probabilistic_peridynamics_gb300 as pp
    from probabilistic_peridynamics_gb300 import integrators
    monkeypatch.setattr(integrators, "cy_worthwhile",
                        lambda *_: route == "pairs")
    n = setup["coords"].shape[0]
    integ = pp.Euler(0.5, fused=route != "functions")
    integ.build(n, 3, setup["nlist"].shape[1], setup["coords"],
                setup["volume"], setup["family"], setup["bc_types"],
                setup["bc_values"], setup["force_bc_types"],
                setup["force_bc_values"], None, None, None)
    z = lambda: np.zeros((n, 3))  # noqa: E731
    integ.create_buffers(setup["nlist"].astype(np.intc).copy(),
                         setup["n_neigh"].astype(np.intc).copy(), 0.05, 0.01,
                         None, z(), z(), z(), z(), z(), np.zeros(n), None, 1,
                         1)
    assert (integ._pairs is not None) == (route == "pairs")
    assert (integ._l0_d is not None) == (route == "break_and_force")
    for t in range(steps):
        if change and t == steps // 2:
            integ.dt, integ.bond_stiffness = 0.25, 0.08
            integ.critical_stretch = 0.008
        integ(4e-3 * (t + 1), 0.05 * (t + 1))
    u, _, _, force, _, damage, nlist, n_neigh = integ.write(
        None, None, None, None, None, None, None, None)
    return u, force, damage, nlist, n_neigh


@pytest.mark.parametrize("change", [False, True])
@pytest.mark.parametrize("form", ["ascending", "shuffled", "twice", "wide"])
@pytest.mark.parametrize("route", ["pairs", "break_and_force"])
def test_same_bits(monkeypatch, route, form, change):
    setup = breaking_lattice() if form == "shuffled" else _setup(form)
    want = _run(monkeypatch, setup, "functions", 40, change)
    got = _run(monkeypatch, setup, route, 40, change)
    for a, b in zip(got, want):
        assert np.array_equal(a, b, equal_nan=True)
    assert int(setup["n_neigh"].sum() - want[4].sum()) > 50  # bonds broke
