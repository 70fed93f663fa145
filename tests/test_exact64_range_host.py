"""The range of the integer route of the bond arithmetic, on the CPU.

``stretch`` (``csrc/pp_exact64.cuh``, which also compiles for the host) leaves
to its caller's function what is outside its range.  Whatever it takes itself
must equal IEEE binary64 arithmetic bit for bit; components that are huge,
infinite or NaN are not its to take, whatever stands beside them, with squares
in integers and with squares by the caller's multiplication.
"""
import ctypes
import itertools
import pathlib
import subprocess

import numpy as np
import pytest

CSRC = (pathlib.Path(__file__).resolve().parent.parent
        / "probabilistic_peridynamics_gb300" / "csrc")

SHIM = """
#include "pp_exact64.cuh"
using namespace pp::exact64;
struct Ops {
    double add(double a, double b) const { return a + b; }
    double mul(double a, double b) const { return a * b; }
};
struct Vec { double x, y, z; };
struct Any {
    int* taken;
    void operator()(double, double, double, double, Stretch* r) const {
        *taken = 0;
        *r = Stretch{0, 0, 0, 0};
    }
};
extern "C" void run(long n, int squares, const double* p, const double* xi,
                    double* out, int* taken) {
    for (long i = 0; i < n; ++i) {
        const Vec v{p[3 * i], p[3 * i + 1], p[3 * i + 2]};
        taken[i] = 1;
        const Any any{taken + i};
        const Stretch r = squares ? stretch<true>(Ops(), v, xi[i], any)
                                  : stretch<false>(Ops(), v, xi[i], any);
        const uint64_t bits[4] = {r.s, r.qx, r.qy, r.qz};
        for (int k = 0; k < 4; ++k) out[4 * i + k] = bits_double(bits[k]);
    }
}
"""

#: Components beyond the range, about its upper end, and ordinary ones.
BEYOND = [2.0 ** 512, 1e155, 1e160, 1e200, 1e300, np.inf, np.nan]
EDGE = [2.0 ** 199, np.nextafter(2.0 ** 201, 0), 2.0 ** 201, 2.0 ** 511,
        2.0 ** -499, 2.0 ** -501, 5e-324]
PLAIN = [0.0, 0.005, -0.005, 3.0, 5.0]


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    folder = tmp_path_factory.mktemp("exact64_range")
    src, so = folder / "shim.cpp", folder / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off",
                    "-shared", "-fPIC", "-I", str(CSRC), str(src), "-o",
                    str(so)], check=True)
    return ctypes.CDLL(str(so))


def _run(shim, p, xi, squares):
    out = np.empty((len(p), 4))
    taken = np.empty(len(p), dtype=np.int32)
    args = [a.ctypes.data_as(ctypes.c_void_p) for a in (p, xi, out, taken)]
    shim.run(ctypes.c_long(len(p)), ctypes.c_int(squares), *args)
    return out, taken.astype(bool)


def _ieee(p, xi):
    with np.errstate(all="ignore"):
        y = np.sqrt(p[:, 0] * p[:, 0] + p[:, 1] * p[:, 1] + p[:, 2] * p[:, 2])
        return np.column_stack([(y - xi) / xi, p / y[:, None]])


@pytest.mark.parametrize("squares", [0, 1])
def test_what_it_takes_is_ieee(shim, squares):
    values = [s * v for v in BEYOND + EDGE for s in (1.0, -1.0)] + PLAIN
    p = np.array(list(itertools.product(values, repeat=3)))
    bad = (~(np.abs(p) < 2.0 ** 201)).any(1)
    for xi in (0.005, 3.0, 5.0, 2.0 ** 199):
        length = np.full(len(p), xi)
        out, taken = _run(shim, p, length, squares)
        assert not (taken & bad).any()
        want = _ieee(p[taken], length[taken])
        assert np.array_equal(out[taken].view(np.uint64),
                              (want + 0.0).view(np.uint64))
        assert taken.any()


@pytest.mark.parametrize("squares", [0, 1])
def test_ordinary_bonds_are_taken(shim, squares):
    rng = np.random.default_rng(5)
    p = rng.normal(size=(100_000, 3)) * 0.005
    xi = np.sqrt((p ** 2).sum(1)) * rng.uniform(0.6, 1.6, len(p))
    out, taken = _run(shim, p, xi, squares)
    assert taken.mean() > 0.99
    assert np.array_equal(out[taken], _ieee(p, xi)[taken])
