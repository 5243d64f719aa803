"""The integer-pipe exponential and logarithms of the land-surface kernels
(pihm-cuda_gb300/csrc/int_math.cuh, compiled for the host: the arithmetic is
integer, so the GPU computes the same bits) against 60-digit references.

Bounds, from the error budgets beside the functions: the exponential within
0.502 ulp; a logarithm within 0.502 ulp where |log2 x| > 1/2 and 0.7 ulp down
to the smallest it takes."""
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
P = ctypes.c_void_p
D = decimal.Decimal


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    so = str(tmp_path_factory.mktemp("im") / "libimel.so")
    subprocess.run([gxx, "-std=c++17", "-O2", "-fPIC", "-shared", "-I", CSRC,
                    os.path.join(HERE, "int_exp_log_host.cpp"), "-o", so], check=True)
    return ctypes.CDLL(so)


def call(f, x, *more):
    x = np.ascontiguousarray(x, np.float64)
    out, ok = np.empty_like(x), np.empty(x.size, np.int32)
    f(P(x.ctypes.data), P(out.ctypes.data), P(ok.ctypes.data), ctypes.c_int64(x.size), *more)
    return out, ok.astype(bool)


def ulps(got, want):
    """|got - want| in units of want's last place (want: Decimal)."""
    u = D(math.ulp(float(want)))
    return float(abs(D(float(got)) - want) / u)


def test_exponential(lib):
    decimal.getcontext().prec = 60
    rng = np.random.default_rng(1)
    x = np.concatenate([rng.uniform(-60.0, 60.0, 1500), rng.uniform(-2.0, 2.0, 1000),
                        rng.choice([-1.0, 1.0], 500) * 2.0 ** rng.uniform(-70.0, 0.0, 500),
                        [0.0, -0.0, 1.0, -1.0, 66.0, -66.0]])
    got, ok = call(lib.im_exp, x)
    assert ok.all()
    assert got[-6] == 1.0 and got[-5] == 1.0
    assert max(ulps(g, D(float(v)).exp()) for g, v in zip(got, x)) < 0.502
    _, ok = call(lib.im_exp, [70.0, -70.0, 1e6, np.inf, -np.inf, np.nan])
    assert not ok.any()


@pytest.mark.parametrize("ten", [0, 1])
def test_logarithm(lib, ten):
    decimal.getcontext().prec = 60
    rng = np.random.default_rng(2 + ten)
    x = np.concatenate([2.0 ** rng.uniform(-120.0, 120.0, 1200), rng.uniform(0.01, 20.0, 1200),
                        2.0 ** (rng.choice([-1.0, 1.0], 600) * rng.uniform(0.02, 0.6, 600))])
    got, ok = call(lib.im_log, x, ctypes.c_int32(ten))
    near = np.abs(np.log2(x)) <= 0.5
    assert ok[np.abs(np.log2(x)) > 2.0 ** -6].all()
    want = [D(float(v)).log10() if ten else D(float(v)).ln() for v in x]
    err = np.array([ulps(g, w) for g, w in zip(got, want)])
    assert err[ok & ~near].max() < 0.502
    assert err[ok & near].max() < 0.7
    _, ok = call(lib.im_log, [1.0, 1.0 + 1e-4, 1.0 - 1e-4, 0.0, -1.0, 5e-324, np.inf, np.nan], ctypes.c_int32(ten))
    assert not ok.any()


@pytest.mark.parametrize("ten", [0, 1])
def test_logarithm_next_to_one(lib, ten):
    decimal.getcontext().prec = 60
    rng = np.random.default_rng(4 + ten)
    d = rng.choice([-1.0, 1.0], 2000) * 2.0 ** rng.uniform(-52.0, -6.01, 2000)
    x = np.concatenate([1.0 + d, [1.0, np.nextafter(1.0, 2.0), np.nextafter(1.0, 0.0)]])
    got, ok = call(lib.im_log_near1, x, ctypes.c_int32(ten))
    assert ok.all()
    assert got[2000] == 0.0
    for g, v in zip(got, x):
        if v != 1.0:
            assert ulps(g, D(float(v)).log10() if ten else D(float(v)).ln()) < 0.502, v
    _, ok = call(lib.im_log_near1, [1.02, 0.98, 2.0, 0.5, 0.0, -1.0, np.inf, np.nan], ctypes.c_int32(ten))
    assert not ok.any()


def cos_ref(x):
    """cos x to 50 digits by its series."""
    x = D(float(x))
    term = s = D(1)
    for k in range(1, 45):
        term *= -x * x / ((2 * k - 1) * (2 * k))
        s += term
    return s


def test_cosine(lib):
    decimal.getcontext().prec = 60
    rng = np.random.default_rng(6)
    x = np.concatenate([3.14 * rng.uniform(0.0, 1.0, 1500), 2.0 ** rng.uniform(-80.0, 0.0, 300),
                        np.pi / 2 + rng.uniform(-1e-3, 1e-3, 200), [0.0, 3.14, 3.1499]])
    got, ok = call(lib.im_cos, x)
    assert ok.all()
    want = [cos_ref(v) for v in x]
    # the absolute error 2^-60 beside the rounding of the result
    for g, w in zip(got, want):
        assert abs(D(float(g)) - w) <= D(math.ulp(float(w))) * D("0.5") + D(2) ** -60, float(w)
    _, ok = call(lib.im_cos, [3.2, 4.0, -1.0, -1e-300, np.inf, np.nan])
    assert not ok.any()
