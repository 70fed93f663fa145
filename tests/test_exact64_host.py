"""The binary64 roots, quotients and squares of ``csrc/pp_exact64.cuh`` on the CPU.

The header also compiles for the host; every result must equal NumPy's
(correctly rounded) ``sqrt`` and division bit for bit, with the FP32 seeds
exact and shifted to either end of the approximation's error bound
(2^-22.9), on random significands, on ones with long runs of zeros and ones,
and on operands built to lie next to a rounding boundary.
"""
import ctypes
import pathlib
import subprocess

import numpy as np
import pytest

CSRC = (pathlib.Path(__file__).resolve().parent.parent
        / "probabilistic_peridynamics_gb300" / "csrc")

SHIM = """
#include "pp_exact64.cuh"
using namespace pp::exact64;
extern "C" void run(long n, float shift, const double* a, const double* b,
                    double* root, double* quotient, double* stretch,
                    double* square, int* fits) {
    seed_shift() = shift;
    for (long i = 0; i < n; ++i) {
        const Divisor y = sqrt_rn(double_bits(a[i] < 0 ? -a[i] : a[i]));
        root[i] = bits_double(pack(y.m, y.e));
        const Divisor d = divisor(double_bits(b[i]));
        quotient[i] = div_signed(double_bits(a[i]), d);
        square[i] = bits_double(square_bits(double_bits(b[i])));
        uint64_t s = 0;
        const Divisor p = divisor(double_bits(a[i] < 0 ? -a[i] : a[i]));
        fits[i] = relative_difference(p, d, s);
        stretch[i] = bits_double(s);
    }
}
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    folder = tmp_path_factory.mktemp("exact64")
    src, so = folder / "shim.cpp", folder / "shim.so"
    src.write_text(SHIM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off",
                    "-shared", "-fPIC", "-I", str(CSRC), str(src), "-o",
                    str(so)], check=True)
    return ctypes.CDLL(str(so))


def _numbers(rng, n, lo, hi):
    """Positive numbers, exponents lo .. hi, significands of every shape."""
    m = rng.integers(0, 1 << 52, n, dtype=np.uint64)
    cut = rng.integers(1, 52, n).astype(np.uint64)
    ones = (np.uint64(1) << cut) - np.uint64(1)
    shape = rng.integers(0, 5, n)
    m = np.where(shape == 1, m & ~ones, m)         # trailing zeros
    m = np.where(shape == 2, m | ones, m)          # trailing ones
    m = np.where(shape == 3, m & np.uint64(63), m)  # just above a power of 2
    m = np.where(shape == 4, ~(m & np.uint64(63)) & np.uint64((1 << 52) - 1),
                 m)                                 # just below
    e = rng.integers(1023 + lo, 1023 + hi + 1, n).astype(np.uint64)
    return (m | (e << np.uint64(52))).view(np.float64)


def _run(shim, a, b, shift):
    a, b = (np.ascontiguousarray(x, dtype=np.float64) for x in (a, b))
    out = [np.empty_like(a) for _ in range(4)]
    fits = np.empty(a.size, dtype=np.int32)
    p = [x.ctypes.data_as(ctypes.c_void_p) for x in (a, b, *out, fits)]
    shim.run(ctypes.c_long(a.size), ctypes.c_float(shift), *p)
    return (*out, fits.astype(bool))


@pytest.mark.parametrize("shift", [0.0, 2.0 ** -22.9, -2.0 ** -22.9])
@pytest.mark.parametrize("case", ["random", "boundary", "near", "zero"])
def test_bits(shim, shift, case):
    rng = np.random.default_rng(11)
    n = 200_000
    b = _numbers(rng, n, -200, 200)
    if case == "random":
        a = _numbers(rng, n, -400, 400) * rng.choice([-1.0, 1.0], n)
    elif case == "boundary":
        # squares of, and products with, numbers a half ulp off
        q = _numbers(rng, n, -100, 100)
        near = np.nextafter(q, np.inf)
        a = np.where(rng.random(n) < 0.5, q * near, near * b)
    elif case == "near":
        a = b * (1.0 + rng.uniform(-1.0, 1.0, n)
                 * 10.0 ** rng.integers(-16, 0, n))
        a = np.abs(a) + 1e-70
    else:
        a = np.zeros(n)
        b[:100] = 1.0
    root, quotient, stretch, square, fits = _run(shim, a, b, shift)
    expect = a / b
    assert np.array_equal(quotient.view(np.uint64), expect.view(np.uint64))
    assert np.array_equal(square.view(np.uint64), (b * b).view(np.uint64))
    if case == "zero":
        return
    expect = np.sqrt(np.abs(a))
    assert np.array_equal(root.view(np.uint64), expect.view(np.uint64))
    expect = ((np.abs(a) - b) / b)[fits] + 0.0
    assert np.array_equal(stretch[fits].view(np.uint64),
                          expect.view(np.uint64))
    if case == "near":
        assert fits.mean() > 0.9
