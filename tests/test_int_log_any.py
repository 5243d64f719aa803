"""The logarithm of the Noah kernels (int_math.cuh, log_any_i), on the host,
against 60-digit references: next to one its series' 0.502 ulp up to the edge
of its range, 0.502 ulp where |log2 x| > 1/2, and between the two 0.59 (two
units of 2^-53 in 1024 log2 x, which is 22.9 at the edge)."""
import ctypes
import decimal
import math
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "pihm-cuda_gb300", "csrc")
P, D = ctypes.c_void_p, decimal.Decimal


@pytest.fixture(scope="module")
def log_any(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    so = str(tmp_path_factory.mktemp("im") / "libimla.so")
    subprocess.run([gxx, "-std=c++17", "-O2", "-fPIC", "-shared", "-I", CSRC,
                    os.path.join(HERE, "int_log_any_host.cpp"), "-o", so], check=True)
    f = ctypes.CDLL(so).im_log_any

    def call(x, ten):
        x = np.ascontiguousarray(x, np.float64)
        out, ok = np.empty_like(x), np.empty(x.size, np.int32)
        f(P(x.ctypes.data), P(out.ctypes.data), P(ok.ctypes.data), ctypes.c_int64(x.size), ctypes.c_int32(ten))
        return out, ok.astype(bool)

    return call


EDGE = 2.0 ** -6


@pytest.mark.parametrize("ten", [0, 1])
@pytest.mark.parametrize("lo,hi,bound", [(1.0 - EDGE, 1.0, 0.502), (1.0, 1.0 + EDGE, 0.502), (0.7, 1.0 - EDGE, 0.59),
                                         (1.0 + EDGE, 1.42, 0.59), (1e-30, 0.7, 0.502), (1.42, 1e30, 0.502)])
def test_error(log_any, lo, hi, bound, ten):
    decimal.getcontext().prec = 60
    x = np.exp(np.random.default_rng(8).uniform(math.log(lo), math.log(hi), 4000))
    x = np.concatenate([x[(x != 1.0)], [v for v in (np.nextafter(lo, 9e99), np.nextafter(hi, 0.0)) if v != 1.0]])
    got, ok = log_any(x, ten)
    assert ok.all()
    for g, v in zip(got, x):
        w = D(float(v)).log10() if ten else D(float(v)).ln()
        assert abs(D(float(g)) - w) < D(bound) * D(math.ulp(float(w))), v


def test_range(log_any):
    for ten in (0, 1):
        got, ok = log_any([1.0, 1.0 - EDGE, 1.0 + EDGE], ten)
        assert ok.all() and got[0] == 0.0
        _, ok = log_any([0.0, -0.0, -1.0, -0.99, 5e-324, np.inf, -np.inf, np.nan], ten)
        assert not ok.any()
