"""Boundary magnitudes that a caller assigns to an ``AdjointProblem`` reach the
pair list's rollout as binary64, whatever their type (no GPU: the library is
replaced), and stay the caller's object."""
import ctypes

import numpy as np
import pytest
import torch

from probabilistic_peridynamics_gb300 import _lib
from tests.adjoint_fake import fake_problem

WANT = [1.0, 2.0, 3.0, 4.0, 5.0, 6.0]


@pytest.mark.parametrize("mags", [
    WANT, tuple(WANT), [1, 2, 3, 4, 5, 6], np.arange(1, 7),
    np.arange(1, 7, dtype=np.float32), torch.arange(1.0, 7.0),
    np.repeat(np.arange(1.0, 7.0), 2)[::2]])
def test_magnitudes(monkeypatch, mags):
    from probabilistic_peridynamics_gb300.adjoint import rollout
    seen = []

    def call(args, pairs, r, *rest):
        values = ctypes.cast(r._obj.mags, ctypes.POINTER(ctypes.c_double))
        seen.append(values[:6])
        return _lib.PP_SUCCESS

    problem = fake_problem(monkeypatch, pp_rollout_forward=call,
                           pp_rollout_backward=call)
    problem.mags = mags
    k = torch.ones(problem.nlist0.shape, dtype=torch.float64,
                   requires_grad=True)
    rollout(k, 0.1, problem, 6, 4).sum().backward()
    assert seen == [WANT, WANT]
    assert problem.mags is mags
    with pytest.raises(IndexError):
        rollout(k, 0.1, problem, len(mags) + 1, 4)
