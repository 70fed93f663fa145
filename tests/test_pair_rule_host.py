"""Whether a run of a known length repays its pair list (no GPU), and that
``Model.simulate`` says the length to the CPU integrator as well."""
import pytest

from probabilistic_peridynamics_gb300 import Euler, pairs


@pytest.mark.parametrize("bonds,below,above", [
    (36_548, 40, 80), (166_508, 20, 40), (418_034, 3, 20),
    (1_025_840, 3, 10), (3_615_952, 3, 10), (10_550_928, 1, 3)])
def test_pairs(monkeypatch, bonds, below, above):
    """Measured calls: slower on pairs up to ``below`` steps, faster from
    ``above``."""
    monkeypatch.setattr(pairs, "fits", lambda *_: True)
    assert not pairs.worthwhile(1000, 128, bonds, None, 1)
    assert not pairs.worthwhile(1000, 128, bonds, None, below)
    assert pairs.worthwhile(1000, 128, bonds, None, above)
    assert pairs.worthwhile(1000, 128, bonds, None, 10_000)
    assert pairs.worthwhile(1000, 128, bonds, None)


@pytest.mark.parametrize("bonds,below,above", [
    (36_548, 5, 10), (166_508, 1, 3), (890_908, 0, 1)])
def test_cpu_integrator(monkeypatch, bonds, below, above):
    monkeypatch.setattr(pairs, "fits", lambda *_: True)
    assert not pairs.cy_worthwhile(1000, 120, bonds, None, below)
    assert pairs.cy_worthwhile(1000, 120, bonds, None, above)
    assert pairs.cy_worthwhile(1000, 120, bonds, None)


def test_what_does_not_fit_is_not_taken(monkeypatch):
    monkeypatch.setattr(pairs, "fits", lambda *_: False)
    assert not pairs.worthwhile(1000, 128, 10 ** 6, None, 1000)
    assert not pairs.cy_worthwhile(1000, 128, 10 ** 6, None, 1000)


def test_the_cpu_integrator_takes_the_length():
    assert Euler(dt=1.0).planned_steps is None
