"""The layout of a mixed-precision run (no GPU): the faster step, and in a near
tie the one whose steps and set-up together are faster over the planned run."""
import types

import pytest

from probabilistic_peridynamics_gb300 import autotune
from tests.test_model_host import HostIntegrator, _model, mesh  # noqa: F401

#: Milliseconds a step: a near tie, a clear gain, a loss of the tiled layout.
TIE = {"tiled/0": 0.095, "tiled/1": 0.099, "untiled/0": 0.097,
       "untiled/2": 0.120}
GAIN = {"tiled/0": 0.130, "tiled/1": 0.124, "untiled/0": 0.190}
LOSS = {"tiled/0": 0.011, "untiled/0": 0.012, "untiled/1": 0.010}


@pytest.mark.parametrize("results,steps,expected", [
    (TIE, 50, "untiled/0"), (TIE, 200, "untiled/0"),
    (TIE, 2000, "untiled/0"),  # 4 ms gained, 5 ms of set-up
    (TIE, 2600, "tiled/0"), (TIE, 20_000, "tiled/0"), (TIE, None, "tiled/0"),
    (GAIN, 50, "tiled/1"), (GAIN, 20_000, "tiled/1"), (GAIN, None, "tiled/1"),
    (LOSS, 50, "untiled/1"), (LOSS, 20_000, "untiled/1"),
    ({"untiled/0": 2.0, "untiled/1": 1.0}, 50, "untiled/1")])
def test_choice(results, steps, expected):
    assert autotune.choose(results, 5.0, steps) == expected


def test_choice_that_is_known(monkeypatch):
    integ = types.SimpleNamespace(
        nnodes=10, max_neighbours=8, _kind=1, stiffness_corrections_d=None,
        bond_types_d=None, node_instance_d=None, compensated=False,
        _may_tile=True, autotune=True, planned_steps=200)
    monkeypatch.setattr(autotune, "_cache", {})
    assert autotune.known_choice(integ) is None  # to be timed
    autotune._cache[autotune._key(integ)] = (TIE, 5.0)
    assert autotune.known_choice(integ) == "untiled/0"
    integ.planned_steps = 20_000
    assert autotune.known_choice(integ) == "tiled/0"
    integ.planned_steps, integ.autotune = 200, False
    assert autotune.known_choice(integ) is None  # as its caller asked


def test_simulate_says_how_long_its_run_is(mesh):  # noqa: F811
    seen = []

    class Planned(HostIntegrator):
        planned_steps = None

        def create_buffers(self, *args):
            seen.append(self.planned_steps)
            super().create_buffers(*args)

    m = _model(mesh, integrator=Planned())
    m.simulate(3)
    m.simulate(5)
    assert seen == [3, 5]
    plain = _model(mesh)
    plain.simulate(3)
    assert not hasattr(plain.integrator, "planned_steps")
