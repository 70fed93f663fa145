"""Plain host work where the library is missing, and host copies of arrays it
is not for (no GPU): NumPy's own results."""
import numpy as np
import pytest

from probabilistic_peridynamics_gb300 import _lib, batch
from tests.test_model_host import _model, mesh  # noqa: F401 (a fixture)


@pytest.fixture
def no_library(monkeypatch, tmp_path):
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", tmp_path / "missing.so")
    with pytest.raises(_lib.LibraryError):
        _lib.lib()


def test_copy_without_the_library(no_library):
    a = np.arange(3_000_000, dtype=np.int64)
    assert a.nbytes > _lib.COPY_BYTES
    b = _lib.host_copy(a)
    assert np.array_equal(a, b) and b.base is None and b is not a


def test_model_without_the_library(no_library, monkeypatch, mesh):  # noqa: F811
    monkeypatch.setattr(_lib, "COPY_BYTES", 1)
    m = _model(mesh)
    out = m.simulate(3)
    assert len(m.integrator.calls) == 3
    for got, held in zip(out[2], m.initial_connectivity):
        assert np.array_equal(got, held) and got is not held


def test_split_without_the_library(monkeypatch, no_library):
    inst = batch.uq_instances(count=3, nx_range=(5, 8), ny_range=(5, 7), nz=3)
    b = batch.concatenate(inst)
    for part, i in zip(b.split(b.nlist, "nlist"), inst):
        assert np.array_equal(part, i.nlist) and part.dtype == np.int64


def test_split_of_narrower_rows():
    """A list trimmed to fewer columns than the instances' own."""
    inst = batch.uq_instances(count=3, nx_range=(5, 8), ny_range=(5, 7), nz=3)
    b = batch.concatenate(inst)
    trimmed = np.ascontiguousarray(b.nlist[:, :5])
    for part, i in zip(b.split(trimmed, "nlist"), inst):
        assert np.array_equal(part, i.nlist[:, :5])
    # fewer rows than nodes: what is there
    few = np.ascontiguousarray(b.nlist[:-2])
    assert np.array_equal(b.split(few, "nlist")[-1], inst[-1].nlist[:-2])


def test_copy_of_objects_and_subclasses(monkeypatch):
    monkeypatch.setattr(_lib, "COPY_BYTES", 1)
    objects = np.array([[1], "two", (3,)] * 2, dtype=object)
    a = _lib.host_copy(objects)
    del objects
    assert a[1] == "two" and a[0] == [1]
    masked = np.ma.masked_array(np.arange(4), mask=[0, 1, 0, 0])
    assert np.array_equal(_lib.host_copy(masked).mask, masked.mask)
    assert _lib.host_copy([1, 2]) == [1, 2]
