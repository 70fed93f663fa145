"""The memory a pair list may take is asked again when its pairs have been
counted (no GPU: the library and the free memory are replaced): a list of
one-sided bonds has twice the pairs that its bonds let expect."""
import ctypes
import types

import pytest

from probabilistic_peridynamics_gb300 import _lib, pairs

MB = 2 ** 20


def _build(monkeypatch, npairs, free, cached):
    asked = []

    def count(args, slot_pair, row_start, scratch, stream):
        n = args._obj.nnodes
        ctypes.cast(row_start, ctypes.POINTER(ctypes.c_int32))[n] = npairs
        return _lib.PP_SUCCESS

    def fill(args, p, row_start, differ, stream):
        ctypes.cast(differ, ctypes.POINTER(ctypes.c_int32))[0] = 0
        return _lib.PP_SUCCESS

    def cached_bytes(device):
        asked.append(1)
        return cached

    monkeypatch.setattr(pairs, "lib", lambda: types.SimpleNamespace(
        pp_pair_count=count, pp_pair_fill=fill))
    monkeypatch.setattr(pairs, "_free_bytes", lambda device: free)
    monkeypatch.setattr(pairs, "_cached_bytes", cached_bytes)
    a = _lib.FusedArgs()
    a.nnodes, a.max_neigh = 1000, 128
    return pairs.DevicePairs.build(a, "cpu", None, 2_000_000), len(asked)


@pytest.mark.parametrize("npairs,free,cached,built,asked", [
    (1_000_000, 0, 0, True, 0),            # listed from both ends
    (2_000_000, 500 * MB, 0, True, 0),     # from one end: 208 MB
    (2_000_000, 300 * MB, 0, False, 1),
    (2_000_000, 300 * MB, 200 * MB, True, 1),
    (1_000_001, 150 * MB, 40 * MB, False, 1),
    (100, 0, 0, True, 0),                  # small
    (2 ** 30, 10 ** 15, 0, False, 0)])
def test_counted_pairs(monkeypatch, npairs, free, cached, built, asked):
    got, queries = _build(monkeypatch, npairs, free, cached)
    assert (got is not None) == built
    assert queries == asked
    if built:
        assert got.struct.npairs == npairs
