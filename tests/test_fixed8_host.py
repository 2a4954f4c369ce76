"""The fixed-point digits of csrc/fixed8.cuh, compiled for the host: bound, cut and the rounded product value over
the whole range of doubles (subnormals, the top binade, overflow), against exact rational arithmetic."""

import ctypes
import math
import os
import random
import shutil
import struct
import subprocess
from fractions import Fraction

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SOURCE = r"""
#include "fixed8.cuh"
extern "C" {
unsigned hi_of(unsigned long long x) { return tincr::cd_hi_bits(x); }
int bound_of(unsigned hi) { return tincr::cd_bound(hi); }
unsigned long long fixed_of(unsigned long long x, int e) { return tincr::cd_fixed_bits<true>(x, e); }
unsigned long long value_of(long long h, long long l, int e) { return tincr::cd_value_any(h, l, e); }
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("fixed8")
    src, so = d / "f.cu", d / "f.so"
    src.write_text(SOURCE)
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O1", "-shared", "-Xcompiler", "-fPIC",
                    "-I", os.path.join(ROOT, "tincr_gb300", "csrc"), str(src), "-o", str(so)], check=True)
    q = ctypes.CDLL(str(so))
    q.hi_of.argtypes, q.hi_of.restype = [ctypes.c_uint64], ctypes.c_uint
    q.bound_of.argtypes = [ctypes.c_uint]
    q.fixed_of.argtypes, q.fixed_of.restype = [ctypes.c_uint64, ctypes.c_int], ctypes.c_uint64
    q.value_of.argtypes, q.value_of.restype = [ctypes.c_int64, ctypes.c_int64, ctypes.c_int], ctypes.c_uint64
    return q


def _bits(x):
    return struct.unpack("<Q", struct.pack("<d", x))[0]


def _double(b):
    return struct.unpack("<d", struct.pack("<Q", b))[0]


def _samples():
    rng = random.Random(1)
    out = [2.0 ** k for k in (-1074, -1073, -1043, -1042, -1041, -1023, -1022, -1, 0, 1, 1000, 1022, 1023)]
    out += [math.nextafter(2.0 ** k, 0.0) for k in (-1040, -1022, -1021, 0, 1, 1000)] + [math.nextafter(math.inf, 0.0)]
    out += [1.96 * (1.0 + s) for s in (-1e-6, -1e-9, 0.0, 1e-9, 1e-6)]
    out += [math.ldexp(rng.uniform(1.0, 2.0), rng.randint(-1074, 1023)) for _ in range(4000)]
    out += [math.ldexp(rng.uniform(1.0, 2.0), rng.randint(-1074, -1020)) for _ in range(2000)]
    return [x for x in out if x > 0.0]


def test_bound_and_cut(lib):
    for x in _samples():
        e = lib.bound_of(lib.hi_of(_bits(x)))
        # |x| 2^(62-E) stays in the range of eight balanced digits, 127/255 2^64
        assert Fraction(x) * Fraction(2) ** (62 - e) <= Fraction(127, 255) * 2 ** 64
        for y in (x, -x, x / 3.0, -x / 1024.0, x * 2.0 ** -40):
            got = (lib.fixed_of(_bits(y), e) - 0x8080808080808080) & (2 ** 64 - 1)
            got -= 2 ** 64 if got >= 2 ** 63 else 0
            assert abs(got - Fraction(y) * Fraction(2) ** (62 - e)) <= Fraction(1, 2)
    assert lib.bound_of(lib.hi_of(_bits(0.0))) == 0
    assert lib.fixed_of(_bits(0.0), 0) == 0x8080808080808080
    for x in (math.inf, -math.inf, math.nan):
        assert lib.bound_of(lib.hi_of(_bits(x))) == 1 << 20


def _rounded(v):
    """The double nearest to the rational v, ties to even, overflow to infinity."""
    try:
        return v.numerator / v.denominator   # correctly rounded, subnormals too
    except OverflowError:
        return math.inf if v > 0 else -math.inf


def test_value_over_the_whole_range(lib):
    rng = random.Random(2)
    for _ in range(20000):
        bits = rng.randint(1, 59)
        h = rng.randint(-2 ** bits, 2 ** bits) if rng.random() < 0.9 else 0
        l = rng.randint(-2 ** 59, 2 ** 59) if rng.random() < 0.5 else rng.randint(-2 ** 20, 2 ** 20)
        e = rng.choice([rng.randint(-2200, 2000), rng.randint(-1180, -1000), rng.randint(900, 1024), rng.randint(-80, 20)])
        got, v = _double(lib.value_of(h, l, e)), Fraction(h * 2 ** 32 + l) * Fraction(2) ** e
        want = _rounded(v)
        if got == want:
            continue
        # of a sum of more than 62 bits the lowest are cut before the rounding: one unit of 2^-61 of it
        assert math.isfinite(want) or abs(v) < Fraction(2) ** 1024 * (1 + Fraction(1, 2 ** 53))
        slack = max(Fraction(2) ** (abs(v).numerator.bit_length() - abs(v).denominator.bit_length() - 52), Fraction(2) ** -1074)   # an ulp
        assert math.isfinite(got) and abs(Fraction(got) - v) <= slack * (Fraction(1, 2) + Fraction(1, 2 ** 7))
