"""An ``AdjointProblem`` on CPU tensors with a library that only records its
calls, for tests of the host side of a rollout."""
import contextlib
import ctypes

import numpy as np
import torch

from probabilistic_peridynamics_gb300 import _lib, adjoint, lattice


class FakeStream:
    def wait_stream(self, other):
        pass


class FakeContext:
    device = "cpu"
    stream = FakeStream()
    stream_handle = ctypes.c_void_p(0)

    def on_stream(self):
        return contextlib.nullcontext()


def fake_problem(monkeypatch, steps=8, **calls):
    """A problem on a pair list; ``calls`` are library functions by name,
    any other returns success."""

    class Library:
        def __getattr__(self, name):
            return calls.get(name, lambda *args: _lib.PP_SUCCESS)

    library = Library()
    monkeypatch.setattr(torch.cuda, "current_stream",
                        lambda *_: FakeContext.stream)
    monkeypatch.setattr(torch.Tensor, "record_stream", lambda *_: None)
    monkeypatch.setattr(adjoint, "lib", lambda: library)
    coords = lattice.lattice_coords(4, 3, 2, 1.0)
    family, nlist, _ = lattice.lattice_family(4, 3, 2, 2.015)
    bonds = int(np.sum(family))

    class Pairs:
        struct = _lib.Pairs(npairs=bonds // 2)

        @classmethod
        def build(cls, *args, **kwargs):
            return cls()

    monkeypatch.setattr(adjoint, "DevicePairs", Pairs)
    bc_types, bc_values = lattice.face_bcs(coords, 0)
    problem = adjoint.AdjointProblem(
        coords, np.ones(len(coords)), nlist, bc_types, bc_values,
        1e-5 * np.arange(1, steps + 1), 0.5, context=FakeContext())
    assert problem.pairs is not None
    return problem
