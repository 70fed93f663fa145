"""The pair form of the binary64 step against the one-kernel form.

``pp_pair_step`` computes each bond once; its results must be those of
``pp_fused_step`` bit for bit for every form of neighbour list and model it
takes: rows of every width, unsorted rows, holes, one-sided entries,
neighbours listed twice, a node listed as its own neighbour, volumes and
corrections that differ between the two ends, bond types with regimes,
instances, breaking bonds, every integrator.
"""
import numpy as np
import pytest

from tests.conftest import cuda_available
from tests.gpu_helpers import breaking_setup, run_integrator

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(),
                                 reason="needs a CUDA GPU")]

FORMS = ["plain", "unsorted", "holes", "one_sided", "twice", "own", "volumes",
         "corrections", "symmetric_corrections", "types", "types_corrections",
         "instances", "wide", "narrow", "row32", "row64", "large"]


def _model(form, kind):
    """(setup, keyword arguments of run_integrator) of one form."""
    rng = np.random.default_rng(3)
    # "large": enough pairs for kernels that let the next one in early
    s = breaking_setup(kind, *((62, 51, 4) if form == "large" else ()))
    n, w = s["nlist"].shape
    nl = s["nlist"].copy()
    more = {}
    if form == "unsorted":
        for i in range(n):
            rng.shuffle(nl[i, :s["family"][i]])
    elif form == "holes":
        nl[rng.random(nl.shape) < 0.2] = -1
    elif form == "one_sided":
        drop = rng.random(nl.shape) < 0.2
        nl[drop & (nl > np.arange(n)[:, None])] = -1
    elif form in ("twice", "own"):
        for i in range(0, n, 3):
            nl[i, s["family"][i]] = i if form == "own" else nl[i, 1]
    elif form == "wide":
        nl = np.concatenate([nl, np.full((n, 512 - w), -1, nl.dtype)], axis=1)
    elif form in ("narrow", "row32", "row64"):
        nl = np.ascontiguousarray(
            nl[:, :{"narrow": 8, "row32": 32, "row64": 64}[form]])
    n, w = nl.shape
    if form == "volumes":
        s["volume"] = s["volume"] * rng.uniform(0.5, 1.5, n)
    if form in ("corrections", "types_corrections"):
        s["stiffness_corrections"] = rng.uniform(0.5, 1.5, nl.shape)
    if form == "symmetric_corrections":
        a = rng.uniform(size=n)
        s["stiffness_corrections"] = 0.5 + (a[:, None] + a[nl]) / 2
    if form.startswith("types"):
        s["bond_types"] = np.where(nl >= 0, rng.integers(0, 2, nl.shape),
                                   0).astype(np.intc)
        k, c = s["k"], s["s0"]
        more = dict(bond_stiffness=np.array([[k, 0.5 * k], [2 * k, k]]),
                    critical_stretch=np.array([[0.5 * c, c], [0.3 * c, c]]),
                    plus_cs=np.array([[0.0, 0.25 * k * c],
                                      [0.0, 0.3 * k * c]]),
                    nregimes=2, nbond_types=2)
    s["nlist"], s["max_neigh"] = nl, w
    s["n_neigh"] = (nl != -1).sum(1).astype(np.intc)
    return s, more


def _run(monkeypatch, form, kind, pairs, steps):
    import probabilistic_peridynamics_gb300 as pp
    from probabilistic_peridynamics_gb300 import integrators
    monkeypatch.setattr(integrators, "worthwhile", lambda *_: pairs)
    s, more = _model(form, kind)
    cls = {"euler": pp.EulerCUDA, "euler_cromer": pp.EulerCromerCUDA,
           "velocity_verlet": pp.VelocityVerletCUDA}[kind]
    integ = cls(dt=s["dt"]) if kind == "euler" else cls(0.5, dt=s["dt"])
    if form == "instances":
        half = (np.arange(s["nnodes"]) >= s["nnodes"] // 2).astype(np.intc)
        integ.set_instances(half, np.array([s["s0"], 0.6 * s["s0"]]))
    out = run_integrator(integ, s, steps, 3e-3 * np.arange(1, steps + 1),
                         force_mags=np.zeros(steps), use_run=True, **more)
    assert (integ._pairs is not None) == pairs
    if pairs and form == "large":
        assert integ._pairs.struct.npairs > 400_000
    return out, s


@pytest.mark.parametrize("form", FORMS)
def test_same_bits(monkeypatch, form):
    one, s = _run(monkeypatch, form, "velocity_verlet", False, 50)
    two, _ = _run(monkeypatch, form, "velocity_verlet", True, 50)
    for a, b in zip(one, two):
        assert np.array_equal(a, b, equal_nan=True)
    assert np.any((one[6] == -1) & (s["nlist"] != -1))  # bonds broke


@pytest.mark.parametrize("kind", ["euler", "euler_cromer"])
def test_integrators(monkeypatch, kind):
    one, _ = _run(monkeypatch, "volumes", kind, False, 50)
    two, _ = _run(monkeypatch, "volumes", kind, True, 50)
    for a, b in zip(one, two):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("width,bonds,expected", [
    (32, 99_999, False), (32, 100_000, True), (33, 1, True),
    (128, 6_818, True), (8, 1000, False), (256, 2 ** 30, False)])
def test_rule(width, bonds, expected):
    import torch
    from probabilistic_peridynamics_gb300.pairs import worthwhile
    assert worthwhile(1000, width, bonds, torch.device("cuda:0")) is expected
