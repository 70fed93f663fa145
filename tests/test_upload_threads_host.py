"""Threads that upload the same host array (no GPU: the library is replaced):
its pages stay locked until no copy reads them."""
import threading
import time
import types

import numpy as np

from probabilistic_peridynamics_gb300 import _lib, integrators


def test_pages_stay_locked_under_a_copy(monkeypatch):
    import torch
    locked, copying, faults = set(), [], []

    def register(address, nbytes):
        if address in locked:
            return _lib.PP_ERROR_CUDA
        locked.add(address)
        return _lib.PP_SUCCESS

    def unregister(address):
        if copying:
            faults.append(address)
        locked.remove(address)
        return _lib.PP_SUCCESS

    library = types.SimpleNamespace(pp_host_register=register,
                                    pp_host_unregister=unregister)
    monkeypatch.setattr(integrators, "lib", lambda: library)
    # (a locked page is pinned memory to torch)
    monkeypatch.setattr(torch.Tensor, "is_pinned",
                        lambda t: t.data_ptr() in locked)

    def slowly(plain):
        def copy(t, *args, **kwargs):
            copying.append(1)
            time.sleep(0.005 * (1 + len(copying)))
            out = plain(t, *args, **kwargs)
            copying.pop()
            return out
        return copy

    monkeypatch.setattr(torch.Tensor, "copy_", slowly(torch.Tensor.copy_))
    monkeypatch.setattr(torch.Tensor, "to", slowly(torch.Tensor.to))
    a = np.random.default_rng(1).random(1 << 20)
    assert a.nbytes >= integrators._REGISTER_BYTES
    threads, out = 4, []
    start = threading.Barrier(threads)

    def work():
        start.wait()
        for _ in range(3):
            out.append(integrators._upload(a, np.float64, "cpu"))

    pool = [threading.Thread(target=work) for _ in range(threads)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    assert len(out) == 3 * threads
    assert all(np.array_equal(t.numpy(), a) for t in out)
    assert faults == [] and not locked
