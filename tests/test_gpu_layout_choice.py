"""One mixed-precision integrator whose layouts nearly tie: untiled for a short
planned run, tiled for a long one, either after the other, with the results of
an integrator of that layout alone."""
import numpy as np
import pytest

from tests.conftest import cuda_available
from tests.gpu_helpers import breaking_setup, run_integrator

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(),
                                 reason="needs a CUDA GPU")]

STEPS = 30


def _run(integ, s, planned):
    integ.planned_steps = planned
    return run_integrator(integ, s, STEPS, 3e-3 * np.arange(1, STEPS + 1))


@pytest.mark.parametrize("corrections", [False, True])
def test_layout_follows_the_planned_run(monkeypatch, corrections):
    import probabilistic_peridynamics_gb300 as pp
    from probabilistic_peridynamics_gb300 import autotune
    monkeypatch.setattr(autotune, "_cache", {})
    monkeypatch.setattr(
        autotune, "_time_layout", lambda integ, tiled, warmup, reps:
        {"tiled/0": 0.097} if tiled else {"untiled/0": 0.098})
    monkeypatch.setattr(autotune, "_time_setup", lambda integ: 5.0)
    s = breaking_setup("velocity_verlet")
    if corrections:
        s["stiffness_corrections"] = np.random.default_rng(1).uniform(
            0.9, 1.1, s["nlist"].shape)
    want = {}
    for tiled in (False, True):
        integ = pp.VelocityVerletCUDA(0.5, dt=s["dt"], precision="mixed",
                                      tiled=tiled, autotune=False)
        want[tiled] = _run(integ, s, None)
        assert (integ.tiling is not None) == tiled
    integ = pp.VelocityVerletCUDA(0.5, dt=s["dt"], precision="mixed")
    for planned, tiled in ((100, False), (20_000, True), (100, False),
                           (None, True), (100, False)):
        got = _run(integ, s, planned)
        assert (integ.tiling is not None) == tiled == integ.tiled
        assert integ.planned_steps is None
        for a, b in zip(got, want[tiled]):
            assert np.array_equal(a, b)
