"""Dot products of FP32 values in the Krylov iterations (csrc/dot_acc.cuh), compiled for the host.

They stand for FP64 sums of the exact products.  Over chains as long as a thread's (one row to some
thousand), with and without cancellation, their error is at most that of the FP64 sum, plus the
rounding of the final result (2^-52 of it) and the last of the some 70 bits kept (2^-65 of the sum
of the magnitudes, five bits left for the length of the chain).
"""
import ctypes
import math
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "waterscapes_gb300", "csrc")

SRC = """
#include "dot_acc.cuh"
extern "C" double dot(int n, const float* a, const float* b) {
    mpet::DotOf<float>::type d;
    for (int i = 0; i < n; ++i) d.add(a[i], b[i]);
    return d.value();
}
"""


@pytest.fixture(scope="module")
def dot(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("dot")
    (d / "d.cpp").write_text(SRC)
    so = str(d / "d.so")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-x", "c++", "-I", CSRC, "-o", so,
                    str(d / "d.cpp")], check=True)
    f = ctypes.CDLL(so).dot
    f.restype = ctypes.c_double
    return lambda a, b: f(len(a), a.ctypes.data_as(ctypes.c_void_p), b.ctypes.data_as(ctypes.c_void_p))


@pytest.mark.parametrize("n", [1, 3, 16, 48, 300, 5000])
@pytest.mark.parametrize("kind", ["random", "cancelling", "scales"])
def test_error_is_below_that_of_an_fp64_sum(dot, n, kind):
    rng = np.random.default_rng(n)
    for _ in range(20):
        a = rng.standard_normal(n).astype(np.float32)
        b = rng.standard_normal(n).astype(np.float32)
        if kind == "cancelling" and n > 1:
            h = n // 2
            a[h:2 * h], b[h:2 * h] = a[:h], -b[:h] * np.float32(1 + 2.0 ** -20)
            p = rng.permutation(n)
            a, b = a[p].copy(), b[p].copy()
        elif kind == "scales":
            a *= (10.0 ** rng.uniform(-12, 6, n)).astype(np.float32)
        pr = a.astype(np.float64) * b.astype(np.float64)  # exact
        exact, mag = math.fsum(pr), math.fsum(np.abs(pr))
        s = 0.0
        for v in pr:
            s += v
        err = abs(dot(a, b) - exact)
        assert err <= abs(s - exact) + 2.0 ** -52 * abs(exact) + 2.0 ** -65 * mag
