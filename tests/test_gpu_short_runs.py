"""Short and long runs of one model through ``Model.simulate``: on one kernel
and on pairs, the same results step for step, and an integrator driven by hand
stays on pairs."""
import numpy as np
import pytest

from tests.conftest import cuda_available
from tests.gpu_helpers import breaking_setup, lattice, run_integrator

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(),
                                 reason="needs a CUDA GPU")]


def _model(tmp_path, integrator):
    import probabilistic_peridynamics_gb300 as pp
    from probabilistic_peridynamics_gb300.mesh import write_vtk
    coords, volume, horizon, _, _, _ = lattice(10, 8, 4, 1.0)
    lo, hi = coords[:, 0].min(), coords[:, 0].max()
    write_vtk(tmp_path / "points.vtk", coords, [])
    return pp.Model(
        tmp_path / "points.vtk", integrator, horizon=horizon,
        critical_stretch=0.02, bond_stiffness=0.01, dimensions=3,
        transfinite=1, volume_total=float(volume.sum()),
        is_displacement_boundary=lambda p: [
            -1.0 if p[0] == lo else 1.0 if p[0] == hi else None, None, None])


@pytest.mark.parametrize("kind,short,long", [("EulerCUDA", 4, 400),
                                             ("Euler", 4, 40)])
def test_routes(tmp_path, kind, short, long):
    import probabilistic_peridynamics_gb300 as pp
    integ = getattr(pp, kind)(dt=0.5)
    m = _model(tmp_path, integ)
    mags = 3e-3 * np.arange(1, long + 1)

    def run(steps, first=1, **state):
        out = m.simulate(steps, first_step=first, write=None,
                         displacement_bc_magnitudes=mags, **state)
        assert integ.planned_steps is None
        return out, integ._pairs is not None

    whole, paired = run(long)
    assert paired
    first, paired = run(short)
    assert not paired
    second, paired = run(long - short, short + 1, u=first[0],
                         connectivity=first[2])
    assert paired
    for i in (0, 1, 3):  # displacement, damage, force
        assert np.array_equal(second[i], whole[i])
    for a, b in zip(second[2], whole[2]):
        assert np.array_equal(a, b)
    assert np.any(whole[1] > 0)


def test_driven_by_hand():
    import probabilistic_peridynamics_gb300 as pp
    s = breaking_setup("euler")
    integ = pp.EulerCUDA(dt=s["dt"])
    run_integrator(integ, s, 2, [1e-3, 2e-3])
    assert integ._pairs is not None
