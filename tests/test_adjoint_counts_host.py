"""Step counts and checkpoint intervals that a rollout takes on a pair list
(no GPU: the library is replaced): integers of any type, and intervals of any
size beyond the number of steps."""
import sys

import numpy as np
import pytest

from probabilistic_peridynamics_gb300 import _lib
from tests.adjoint_fake import fake_problem


@pytest.mark.parametrize("steps,every,expected", [
    (8, 3, (8, 3)), (np.int64(8), 3, (8, 3)), (8, np.int32(3), (8, 3)),
    (8, 8, (8, 8)), (8, 2 ** 31, (8, 8)), (8, sys.maxsize, (8, 8)),
    (8, 10 ** 30, (8, 8)), (0, 5, (0, 1)), (True, 5, (1, 1))])
def test_counts(monkeypatch, steps, every, expected):
    import torch
    from probabilistic_peridynamics_gb300.adjoint import rollout
    seen = []

    def call(args, pairs, r, *rest):
        seen.append((r._obj.steps, r._obj.every))
        return _lib.PP_SUCCESS

    problem = fake_problem(monkeypatch, pp_rollout_forward=call,
                           pp_rollout_backward=call)
    k = torch.ones(problem.nlist0.shape, dtype=torch.float64,
                   requires_grad=True)
    rollout(k, 0.1, problem, steps, every).sum().backward()
    assert seen == [expected, expected]


@pytest.mark.parametrize("steps,every", [(8, 0), (8, -3), (8, 3.0),
                                         (8.0, 3), (-1, 3)])
def test_others_stay_on_the_single_steps(monkeypatch, steps, every):
    import torch
    from probabilistic_peridynamics_gb300.adjoint import rollout
    calls = []
    problem = fake_problem(
        monkeypatch, pp_rollout_forward=lambda *_: calls.append(1),
        pp_fused_step=lambda *_: _lib.PP_SUCCESS)
    k = torch.ones(problem.nlist0.shape, dtype=torch.float64)
    try:
        rollout(k, 0.1, problem, steps, every)
    except (TypeError, ZeroDivisionError):
        pass
    assert calls == []
