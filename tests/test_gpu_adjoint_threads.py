"""Two host threads with one ``AdjointProblem``: states and gradients are those
of the same rollouts one after the other, bit for bit."""
import threading

import numpy as np
import pytest

from tests.conftest import cuda_available

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not cuda_available(),
                                 reason="needs a CUDA GPU")]


def test_two_threads():
    import torch
    from probabilistic_peridynamics_gb300 import lattice
    from probabilistic_peridynamics_gb300.adjoint import (AdjointProblem,
                                                          rollout)
    steps, every, repeats = 60, 7, 4
    coords = lattice.lattice_coords(12, 10, 5, 1.0)
    _, nlist, _ = lattice.lattice_family(12, 10, 5, 3.015)
    bc_types, bc_values = lattice.face_bcs(coords, 0, tol=0.3)
    prob = AdjointProblem(coords, np.ones(len(coords)), nlist, bc_types,
                          bc_values, 1e-5 * np.arange(1, steps + 1), 0.5)
    assert prob.pairs is not None

    def run(scale):
        k = torch.full(nlist.shape, 0.01 * scale, dtype=torch.float64,
                       device="cuda", requires_grad=True)
        u = rollout(k, 0.03, prob, steps, every)
        (u ** 2).sum().backward()
        return u.detach().cpu().numpy(), k.grad.cpu().numpy()

    want = [run(1.0), run(1.3)]
    got = [[], []]
    start = threading.Barrier(2)

    def work(w):
        start.wait()
        for _ in range(repeats):
            got[w].append(run((1.0, 1.3)[w]))

    pool = [threading.Thread(target=work, args=(w,)) for w in range(2)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    for w in range(2):
        assert len(got[w]) == repeats
        for u, g in got[w]:
            assert np.array_equal(u, want[w][0])
            assert np.array_equal(g, want[w][1])
