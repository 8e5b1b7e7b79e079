"""Sums of the one-launch Gram-Schmidt (csrc/longsum.cuh), compiled for the host: the FP32 form against exact
arithmetic on as many products as a thread of the largest mesh adds, and on a warp's tree of them."""
import ctypes
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "earthbyte_underworld_gb300", "csrc")
SOURCE = """
#include "longsum.cuh"
extern "C" double warp_sum(int n, const float* a, const float* b) {
    uwg::LongSum<float> lane[32];
    for (int i = 0; i < n; ++i) lane[i % 32].add(a[i], b[i]);
    for (int o = 16; o > 0; o >>= 1)
        for (int k = 0; k < o; ++k) lane[k].merge(lane[k + o]);
    return lane[0].value();
}
"""


@pytest.fixture(scope="module")
def warp_sum(tmp_path_factory):
    d = tmp_path_factory.mktemp("longsum")
    (d / "s.cpp").write_text(SOURCE)
    subprocess.run([shutil.which("g++"), "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "s.cpp"), "-o",
                    str(d / "s.so")], check=True)
    f = ctypes.CDLL(str(d / "s.so")).warp_sum
    f.restype = ctypes.c_double
    f.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
    return lambda a, b: f(len(a), a.ctypes.data, b.ctypes.data)


@pytest.mark.parametrize("n", [1, 31, 33, 59 * 32, 118 * 32 + 7])
@pytest.mark.parametrize("kind", ["equal", "positive", "mixed", "wide"])
def test_sum_of_rounded_products(warp_sum, n, kind):
    rng = np.random.default_rng(n)
    a = {"equal": np.full(n, 0.1), "positive": rng.uniform(0.5, 1.0, n), "mixed": rng.standard_normal(n),
         "wide": rng.standard_normal(n) * 10.0 ** rng.uniform(-12, 12, n)}[kind].astype(np.float32)
    b = (a if kind in ("equal", "positive") else rng.permutation(a)).copy()
    p = a * b   # each product is rounded once, as a single FP32 product per thread is
    exact = sum(map(Fraction, p.tolist()))
    size = sum(abs(Fraction(v)) for v in p.tolist())
    # a pair's low part is rounded once or twice per addition: n additions of 2^-48 of the sum of magnitudes
    assert abs(Fraction(warp_sum(a, b)) - exact) <= Fraction(n) * size / 2 ** 47
    if kind == "equal" and n == 59 * 32:   # what a plain chain of 59 and a tree lose on the same values
        chain = np.float32(0)
        for _ in range(59):
            chain = np.float32(chain + p[0])
        assert abs(Fraction(float(chain)) * 32 - exact) > exact / 2 ** 21


def test_not_finite(warp_sum):
    big, nan = np.full(64, 1e30, np.float32), np.full(64, np.nan, np.float32)
    assert warp_sum(big, big) == np.inf and np.isnan(warp_sum(nan, big))
