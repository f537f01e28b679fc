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
