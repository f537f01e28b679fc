"""The device's own arithmetic against exact values.

Small kernels (device_arithmetic.cu) apply the functions of the solver's
headers to arrays; the expected values are exact rationals, rounded here.
"""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    from doug_gb300 import build as B
    so = str(tmp_path_factory.mktemp("arith") / "device_arithmetic.so")
    subprocess.run([B._nvcc(), B.ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-I", B.CSRC,
                    "-o", so, os.path.join(HERE, "device_arithmetic.cu")], check=True)
    return ctypes.CDLL(so)


def _p(a):
    return ctypes.c_void_p(a.ctypes.data)


def test_split_value_is_the_rounded_sum(lib):
    """sum_s d_s 2^(8 (7 - s)) 2^(ex - 2112): within half a unit in the last
    place of the result (the last subnormal place below the normal numbers;
    a tie goes either way), infinity from the rounding limit of the largest
    number on."""
    rng = np.random.default_rng(1)
    n = 40000
    d = (rng.integers(-(1 << 24), (1 << 24) + 1, (n, 8)) >> rng.integers(0, 25, (n, 8))).astype(np.int32)
    d[rng.random((n, 8)) < 0.3] = 0
    d[:8] = 0
    ex = rng.integers(2, 4093, n).astype(np.int32)
    near = rng.integers(0, n, n // 2)
    ex[near[: n // 4]] = rng.integers(950, 1090, n // 4)  # around the smallest normal numbers
    ex[near[n // 4:]] = rng.integers(3040, 3130, n // 4)  # and the largest
    out = np.zeros(n)
    assert lib.split_value(n, _p(d), _p(ex), _p(out)) == 0
    seen = {"sub": 0, "top": 0, "inf": 0, "zero": 0}
    limit = Fraction(2) ** 1024 - Fraction(2) ** 970  # rounds to infinity from here on
    for i in range(n):
        v = sum(int(d[i, s]) << (8 * (7 - s)) for s in range(8)) * Fraction(2) ** (int(ex[i]) - 2112)
        if abs(v) >= limit:
            assert np.isinf(out[i]) and (out[i] > 0) == (v > 0)
            seen["inf"] += 1
            continue
        got = Fraction(float(out[i]))
        ulp = Fraction(float(np.spacing(abs(out[i]))))
        assert abs(got - v) <= ulp / 2
        seen["zero"] += got == 0
        seen["sub"] += 0 < abs(got) < Fraction(2) ** -1022
        seen["top"] += abs(got) >= Fraction(2) ** 1023
    assert min(seen.values()) > 50


def _pivots(dtype, n):
    """Positive numbers over the whole range, subnormal ones too, and its ends."""
    rng = np.random.default_rng(2)
    info = np.finfo(dtype)
    e = rng.integers(info.minexp - info.nmant, info.maxexp, n)
    d = np.ldexp(rng.uniform(1.0, 2.0, n), e).astype(dtype)
    d[:6] = [info.tiny, info.max, np.nextafter(info.tiny, 0), np.ldexp(1.0, info.minexp - info.nmant), 1.0,
             np.nextafter(dtype(2), dtype(0))]
    # around the powers of two where a pivot is kept in another way
    d[6:60] = np.ldexp(rng.uniform(1.0, 1.99, 54), rng.integers(info.maxexp - 4, info.maxexp, 54)).astype(dtype)
    d[60:120] = np.ldexp(rng.uniform(1.0, 2.0, 60), rng.integers(info.minexp - 3, info.minexp + 3, 60)).astype(dtype)
    return np.maximum(d, np.ldexp(1.0, info.minexp - info.nmant).astype(dtype))


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_pivots(lib, dtype):
    """Reciprocal: within half a unit in the last place and 2^-10 of one (the
    FP64 iteration's error is 2^-63 before its rounding).  Quotient: two
    roundings, 2^-nmant relative (and 2^-10 of it for the reciprocal's), or half a
    unit of the last subnormal place more.  Root: the reciprocal's rounding halved, those of root, division and
    product: 2^-nmant relative (always a normal number)."""
    n = 6000
    info = np.finfo(dtype)
    d = _pivots(dtype, n)
    rng = np.random.default_rng(3)
    with np.errstate(over="ignore"):
        c = (rng.uniform(-1, 1, n) * np.sqrt(d.astype(np.longdouble))).astype(dtype)  # an entry of L times a root
    inv, quot, root = (np.zeros(n, dtype) for _ in range(3))
    assert getattr(lib, "pivot_f64" if dtype == np.float64 else "pivot_f32")(n, *map(_p, (c, d, inv, quot, root))) == 0
    rel, sub = Fraction(2) ** -info.nmant, Fraction(2) ** (info.minexp - info.nmant)
    top = Fraction(float(info.max))
    for i in range(n):
        x, num = Fraction(float(d[i])), Fraction(float(c[i]))
        if 1 / x < top:
            ulp = Fraction(float(np.spacing(inv[i])))
            assert abs(Fraction(float(inv[i])) - 1 / x) <= ulp * (Fraction(1, 2) + Fraction(1, 1024))
        assert abs(Fraction(float(quot[i])) - num / x) <= rel * Fraction(1025, 1024) * abs(num / x) + sub
        r = Fraction(float(root[i]))  # r^2 x = 1 to twice the relative error
        assert abs(r * r * x - 1) <= 2 * rel + rel * rel


def test_widening_is_exact(lib):
    x = np.random.default_rng(4).integers(0, 1 << 32, 2_000_000, dtype=np.uint64).astype(np.uint32)
    x[:8] = [0, 0x80000000, 1, 0x007fffff, 0x00800000, 0x7f7fffff, 0x7f800000, 0xff800000]
    f = x.view(np.float32)
    y = np.zeros(len(f))
    assert lib.widen(len(f), _p(f), _p(y)) == 0
    with np.errstate(invalid="ignore"):
        ref = f.astype(np.float64)
    assert np.array_equal(y, ref, equal_nan=True) and np.array_equal(np.signbit(y), np.signbit(ref) | (np.isnan(y) & np.signbit(y)))


def test_narrowing_rounds_to_nearest_even(lib):
    rng = np.random.default_rng(5)
    n = 2_000_000
    x = rng.integers(0, 1 << 63, n, dtype=np.uint64) | (rng.integers(0, 2, n, dtype=np.uint64) << np.uint64(63))
    e = rng.integers(896 - 30, 1152, n).astype(np.uint64)  # most around what FP32 holds
    near = rng.random(n) < 0.9
    x[near] = (x[near] & np.uint64(0x800fffffffffffff)) | (e[near] << np.uint64(52))
    tie = rng.random(n) < 0.3  # halfway between two numbers, or a bit beside it
    x[tie] = (x[tie] & np.uint64(0xffffffffe0000000)) | np.uint64(0x10000000)
    side = tie & (rng.random(n) < 0.5)
    x[side] += rng.integers(-1, 2, side.sum()).astype(np.int64).view(np.uint64)
    x[:6] = [0, 1 << 63, 1, 0x7ff0000000000000, 0xfff0000000000000, 0x7fefffffffffffff]
    d = x.view(np.float64)
    y = np.zeros(n, np.float32)
    assert lib.narrow(n, _p(d), _p(y)) == 0
    with np.errstate(over="ignore", invalid="ignore"):
        ref = d.astype(np.float32)
    assert np.array_equal(y, ref, equal_nan=True)
    assert np.array_equal(np.signbit(y[~np.isnan(ref)]), np.signbit(ref[~np.isnan(ref)]))
