"""The short fp32 sums that stand for 64-bit ones in the likelihood's per-epoch passes (pg_sums.cuh), compiled for
the host, against exact rational sums: sums of up to 32 weights, and of weights times features, are the exact
sum rounded to 64 bits (2^-53 of it, and 2^-60 of the terms' magnitudes where they cancel)."""
import ctypes as C
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

from paragraph_gb300.build import ROOT, nvcc


@pytest.fixture(scope="module")
def sums(tmp_path_factory):
    so = tmp_path_factory.mktemp("sums") / "libsums.so"
    cuda = Path(nvcc()).resolve().parents[1] / "include"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-I", str(cuda), "-o", str(so),
                    str(ROOT / "tests" / "sums_host.cpp")], check=True)
    lib = C.CDLL(str(so))
    lib.sum_values.restype = lib.sum_products.restype = C.c_double
    lib.sum_values.argtypes = [C.c_void_p, C.c_int, C.POINTER(C.c_int)]
    lib.sum_products.argtypes = [C.c_void_p, C.c_void_p, C.c_int]
    return lib


def _exact(terms):
    return sum(terms, Fraction(0)), sum((abs(t) for t in terms), Fraction(0))


def _frac(a):
    return [Fraction(float(x)) for x in a]


@pytest.mark.parametrize("spread", [0, 2, 12, 30, 60])
@pytest.mark.parametrize("n", [1, 2, 3, 31, 32])
def test_sums_are_64_bit_sums(sums, n, spread):
    rng = np.random.default_rng(100 * n + spread)
    holds = C.c_int()
    for trial in range(200):
        top = rng.uniform(-50, 90 - 5)
        w = ((1.0 + rng.random(n)) * 2.0 ** (top - rng.uniform(0, spread, n) - 1)).astype(np.float32)
        got = sums.sum_values(w.ctypes.data, n, C.byref(holds))
        want, _ = _exact(_frac(w))
        assert abs(Fraction(got) - want) <= want * Fraction(1, 2**53) * Fraction(1001, 1000)
        assert holds.value == (2.0**-60 <= got <= 2.0**90)
        if not holds.value:
            continue
        # ages, logarithms of degrees and of fitness values, of either sign
        f = [np.round(rng.random(n) * 10.0 ** rng.uniform(0, 9)), np.log1p(np.floor(10.0 ** rng.uniform(0, 6, n))),
             rng.normal(0.0, 1.0, n)][trial % 3].astype(np.float32)
        got = sums.sum_products(w.ctypes.data, f.ctypes.data, n)
        want, size = _exact([a * b for a, b in zip(_frac(w), _frac(f))])
        assert abs(Fraction(got) - want) <= abs(want) * Fraction(1001, 1000 * 2**53) + size * Fraction(1, 2**60)


def test_ranges_that_do_not_hold_are_known(sums):
    holds = C.c_int()
    for w, ok in (([0.0] * 32, 1), ([2.0**-61], 0), ([2.0**-60], 1), ([2.0**-60, 2.0**-140], 1), ([2.0**90], 1),
                  ([2.0**90, 2.0**90], 0), ([3e38] * 32, 0), ([float("inf")], 0), ([float("nan")], 0), ([1e-45], 0)):
        a = np.array(w, np.float32)
        sums.sum_values(a.ctypes.data, len(a), C.byref(holds))
        assert holds.value == ok, w
