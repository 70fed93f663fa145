"""Rollouts of several threads on one ``AdjointProblem`` queue their launches
one call after the other (no GPU): the calls release the interpreter lock,
and the force records of the problem's pair list pass from one kernel of a
step to the next."""
import threading
import time

from probabilistic_peridynamics_gb300 import _lib
from tests.adjoint_fake import fake_problem


def test_one_thread_queues_at_a_time(monkeypatch):
    import torch
    inside, overlaps, calls = [], [], []

    def queue(*args):
        inside.append(1)
        time.sleep(0.02)
        overlaps.append(len(inside) > 1)
        inside.pop()
        calls.append(1)
        return _lib.PP_SUCCESS

    problem = fake_problem(monkeypatch, pp_rollout_forward=queue,
                           pp_rollout_backward=queue)
    k = torch.ones(problem.nlist0.shape, dtype=torch.float64)
    threads = 4
    start = threading.Barrier(threads)

    def work():
        start.wait()
        u, checkpoints, breaks = problem.run_forward(k, 8, 3, 0.1)
        problem.run_backward(u, k, 8, 3, checkpoints, breaks)

    pool = [threading.Thread(target=work) for _ in range(threads)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    assert len(calls) == 2 * threads
    assert not any(overlaps)
