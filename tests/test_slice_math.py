"""Digits, magnitudes and recombination of the sliced FP64 GEMM (slice_math.cuh) on the host:
the header is compiled with the host compiler and checked against exact arithmetic."""
import ctypes
import math
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "slice_math.cuh"
using namespace scess;
extern "C" {
int64_t fixed(double x, int e) { return slice_fixed(x, e); }
int digit(int64_t f, int p) { return slice_digit(f + kDigitBias, p); }
double value(int64_t t, int w, int fs, int sc, uint32_t flip) { return slice_value(t, w, fs, sc, flip); }
unsigned magnitude(double x, int e) { return slice_magnitude(x, e); }
}
"""


@pytest.fixture(scope='module')
def lib(tmp_path_factory):
    cxx = shutil.which('g++')
    if not cxx:
        pytest.skip('no host compiler')
    d = tmp_path_factory.mktemp('slice_math')
    (d / 'm.cpp').write_text(SOURCE)
    so = d / 'm.so'
    subprocess.run([cxx, '-std=c++17', '-O2', '-shared', '-fPIC', '-I', os.path.join(ROOT, 'scess_gb300', 'csrc'),
                    str(d / 'm.cpp'), '-o', str(so)], check=True)
    m = ctypes.CDLL(str(so))
    m.fixed.restype = ctypes.c_int64
    m.fixed.argtypes = [ctypes.c_double, ctypes.c_int]
    m.digit.argtypes = [ctypes.c_int64, ctypes.c_int]
    m.value.restype = ctypes.c_double
    m.value.argtypes = [ctypes.c_int64, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_uint32]
    m.magnitude.restype = ctypes.c_uint
    m.magnitude.argtypes = [ctypes.c_double, ctypes.c_int]
    return m


def biased(x):
    return int(np.float64(x).view(np.uint64) >> np.uint64(52)) & 0x7ff


def values(rng, n):
    x = rng.standard_normal(n) * 2.0**rng.integers(-70, 1, n)
    return np.concatenate([x, [0.0, 1.0, -1.0, 1.0 - 2.0**-53, -(1.0 - 2.0**-53), 2.0**-1060, 2.0**-1022]])


def test_digits_add_up_to_the_value(lib):
    rng = np.random.default_rng(0)
    for x in values(rng, 2000):
        for up in (0, 1, 9, 40):
            e = max(biased(x), 1) + up  # the row's largest exponent
            f = lib.fixed(x, e)
            d = [lib.digit(f, p) for p in range(7)]
            assert abs(d[0]) <= 64 and all(-256 <= v <= 255 for v in d[1:])
            assert sum(v * 512**(6 - p) for p, v in enumerate(d)) == f
            exact = Fraction(float(x)) * Fraction(2)**(60 - (e - 1022))
            assert abs(exact - f) <= Fraction(1, 2)
            if up <= 7 and biased(x):
                assert exact == f  # (within 2^-7 of the row's largest: no rounding)


def test_magnitudes_are_rounded_down_and_never_vanish(lib):
    rng = np.random.default_rng(1)
    for x in values(rng, 2000):
        for up in (0, 5, 58, 59, 300):
            e = max(biased(x), 1) + up
            m = np.uint32(lib.magnitude(x, e) << 16).view(np.float32)
            rel = abs(Fraction(float(x))) * Fraction(2)**(1022 - e)
            if x == 0.0:
                assert m == 0.0
            elif rel < Fraction(2)**-60 or biased(x) == 0:
                assert m == np.float32(2.0**-60)
            else:
                assert Fraction(float(m)) <= max(rel, Fraction(2)**-60) and Fraction(float(m)) * 129 >= rel * 128


def test_values_are_rounded_to_nearest(lib):
    rng = np.random.default_rng(2)
    for _ in range(4000):
        t = int(rng.integers(-2**62, 2**62)) >> int(rng.integers(0, 62))
        fs = int(rng.integers(6, 21))
        w = int(rng.integers(-2**30, 2**30)) >> int(rng.integers(0, 30))
        sc = int(rng.integers(-900, 800))
        got = lib.value(t, w, fs, sc, 0)
        exact = (Fraction(t) + Fraction(w, 2**fs)) * Fraction(2)**sc
        want = exact.numerator / exact.denominator  # (correctly rounded)
        assert got == want or abs(got - want) <= math.ulp(want) and tie(exact)
        assert lib.value(t, w, fs, sc, 0x80000000) == (-got if got else 0.0)


def tie(x):
    """Halfway between two doubles: rounded up in magnitude here, to even by IEEE."""
    x = abs(x)
    e = x.numerator.bit_length() - x.denominator.bit_length()
    scaled = x * Fraction(2)**(60 - e)
    while scaled >= 2**53:
        scaled /= 2
    while scaled < 2**52:
        scaled *= 2
    return scaled.denominator == 2


@pytest.mark.parametrize('sc', [-1500, -1100, -1074, -1030, 970, 1020, 1100])
def test_values_beyond_the_normal_numbers(lib, sc):
    for t in (1, 3, -5, (1 << 40) + 1, -(1 << 61) + 12345):
        got = lib.value(t, 0, 20, sc, 0)
        try:
            want = math.ldexp(float(t), sc)
        except OverflowError:
            want = math.copysign(math.inf, t)
        assert got == want or abs(got - want) <= 5e-324  # (two roundings below the normal numbers)
