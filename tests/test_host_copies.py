"""Threaded host copies of the library (no GPU): equal to NumPy's at sizes on
either side of a piece, with a remainder, and with strided and other arrays."""
import ctypes

import numpy as np
import pytest

from probabilistic_peridynamics_gb300 import _lib, batch


@pytest.mark.parametrize("size", [0, 1, (4 << 20) - 1, (8 << 20) + 3,
                                  (33 << 20) + 5])
def test_copy(size):
    a = np.random.default_rng(1).integers(0, 255, size, dtype=np.uint8)
    assert np.array_equal(_lib.host_copy(a), a)
    b = np.zeros_like(a)
    assert _lib.lib().pp_host_copy(b.ctypes.data, a.ctypes.data, size) == 0
    assert np.array_equal(a, b)


def test_copy_of_other_layouts():
    a = np.arange(3_000_000.0).reshape(1000, 3000)
    for x in (a.T, a[::2], np.asfortranarray(a)):
        c = _lib.host_copy(x)
        assert np.array_equal(c, x) and c.flags.c_contiguous
        assert c.dtype == x.dtype and c.base is None


@pytest.mark.parametrize("rows,width,columns", [(0, 8, 8), (1, 1, 1),
                                                (5, 128, 64),
                                                (40_001, 32, 32),
                                                (9_999, 64, 64)])
def test_local_rows(rows, width, columns):
    rng = np.random.default_rng(2)
    src = rng.integers(-1, 100, (rows, width), dtype=np.int32) + 0
    src = np.where(src >= 0, src + 2 ** 30, -1).astype(np.int32)
    dst = np.full((rows, columns), 7, dtype=np.int64)
    assert _lib.lib().pp_host_local_rows(
        src.ctypes.data_as(ctypes.c_void_p), rows, width, columns, 2 ** 30,
        dst.ctypes.data_as(ctypes.c_void_p)) == 0
    want = np.where(src[:, :columns] >= 0,
                    src[:, :columns] - np.int64(2 ** 30), -1)
    assert np.array_equal(dst, want)


def test_split_rows_as_numpy_gives_them():
    inst = batch.uq_instances(count=3, nx_range=(5, 8), ny_range=(5, 7), nz=3)
    b = batch.concatenate(inst)
    for k, part in enumerate(b.split(b.nlist, "nlist")):
        a, e = b.offsets[k], b.offsets[k + 1]
        w = inst[k].nlist.shape[1]
        rows = b.nlist[a:e]
        want = np.where(rows[:, :w] >= 0, rows[:, :w] - a, -1)
        assert np.array_equal(part, want) and part.dtype == want.dtype
    for x, y in zip(b.split(b.nlist, "nlist"),
                    b.split(np.asfortranarray(b.nlist), "nlist")):
        assert np.array_equal(x, y) and x.dtype == y.dtype
