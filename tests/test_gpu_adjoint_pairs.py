"""The rollout on a pair list against the step-by-step rollout.

The forward states are the same bit for bit.  The gradients come from other
operations (reciprocals instead of divisions, fused multiply-adds, sums of
pairs): each bond's reverse step differs by about fifty binary64 roundings and
accumulates over the steps, 50 * 1.1e-16 * 40 = 2e-13 of the largest gradient
here, so 1e-11 is asked for.  A list with a one-sided bond keeps the
step-by-step route.
"""
import numpy as np
import pytest

from tests.conftest import cuda_available

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(),
                                 reason="needs a CUDA GPU")]

STEPS = 40


def _problem(form):
    from probabilistic_peridynamics_gb300 import lattice
    from probabilistic_peridynamics_gb300.adjoint import AdjointProblem
    rng = np.random.default_rng(4)
    coords = lattice.lattice_coords(7, 6, 4, 1.0)
    _, nlist, _ = lattice.lattice_family(7, 6, 4, 3.015)
    n = len(coords)
    if form == "jittered":
        coords = coords + rng.uniform(-0.1, 0.1, coords.shape)
    if form == "one_sided":
        nlist[n // 2, 0] = -1
    bc_types, bc_values = lattice.face_bcs(coords, 0, tol=0.3)
    volume = rng.uniform(0.8, 1.2, n)
    rate = 2e-3 if form == "breaks" else 1e-5
    prob = AdjointProblem(coords, volume, nlist, bc_types, bc_values,
                          rate * np.arange(1, STEPS + 1), 0.5)
    k = np.where(nlist != -1, 0.01 * rng.uniform(0.9, 1.1, nlist.shape), 0.0)
    return prob, k


def _run(prob, k, every):
    import torch
    from probabilistic_peridynamics_gb300.adjoint import rollout
    kt = torch.tensor(k, dtype=torch.float64, device="cuda",
                      requires_grad=True)
    u = rollout(kt, 0.03, prob, STEPS, every)
    (u ** 2).sum().backward()
    return u.detach().cpu().numpy(), kt.grad.cpu().numpy()


@pytest.mark.parametrize("form,every", [("elastic", 7), ("elastic", 1),
                                        ("elastic", 100), ("jittered", 10),
                                        ("breaks", 7), ("breaks", 40),
                                        ("one_sided", 7)])
def test_pair_rollout(form, every):
    prob, k = _problem(form)
    assert (prob.pairs is None) == (form == "one_sided")
    u1, g1 = _run(prob, k, every)
    prob.pairs = None
    u2, g2 = _run(prob, k, every)
    assert np.array_equal(u1, u2)
    assert np.abs(g1 - g2).max() <= 1e-11 * np.abs(g2).max()
    assert np.abs(g2).max() > 0
