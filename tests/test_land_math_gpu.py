"""The land-surface step's exponential and logarithm against 60-digit
references.  Both are 0.502 ulp functions with a rounding beside them of the
double-double routines' 2^-62 of the result, so 0.52 ulp holds everywhere:
where the fixed-point logarithm is not that close (0.7 to 1.42), next to one,
and where the fixed-point exponential ends (66.5)."""
import ctypes
import decimal
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
D = decimal.Decimal
BOUND = 0.52


def _run(x):
    import torch

    from pihm_gpu import capi
    f = capi.load().pihm_gpu_selftest_land_exp_log
    f.argtypes = [ctypes.c_void_p] * 3 + [ctypes.c_int64, ctypes.c_void_p]
    a = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    e, l = torch.empty_like(a), torch.empty_like(a)
    assert f(a.data_ptr(), e.data_ptr(), l.data_ptr(), a.numel(), None) == 0
    torch.cuda.synchronize()
    return e.cpu().numpy(), l.cpu().numpy()


def _worst(got, want):
    return max(float(abs(D(float(g)) - w) / D(math.ulp(float(w)))) for g, w in zip(got, want))


@pytest.mark.parametrize("lo,hi", [(0.7, 0.985), (1.015, 1.42), (0.69, 0.71), (1.41, 1.43), (0.984, 1.016),
                                   (1e-3, 0.7), (1.42, 1e4)])
def test_logarithm(lo, hi):
    decimal.getcontext().prec = 60
    x = np.exp(np.random.default_rng(3).uniform(math.log(lo), math.log(hi), 3000))
    assert _worst(_run(x)[1], [D(float(v)).ln() for v in x]) < BOUND


@pytest.mark.parametrize("lo,hi", [(-5.0, 5.0), (-70.0, 70.0), (66.0, 68.0), (-690.0, -66.0), (66.0, 690.0)])
def test_exponential(lo, hi):
    decimal.getcontext().prec = 60
    x = np.random.default_rng(4).uniform(lo, hi, 3000)
    assert _worst(_run(x)[0], [D(float(v)).exp() for v in x]) < BOUND


def test_special_values():
    e, l = _run(np.array([0.0, -0.0, 1.0, np.inf, -np.inf, np.nan, -1.0, 5e-324, 710.0, -750.0]))
    assert e[0] == e[1] == 1.0 and e[3] == np.inf and e[4] == 0.0 and np.isnan(e[5]) and e[8] == np.inf and e[9] == 0.0
    assert l[0] == l[1] == -np.inf and l[2] == 0.0 and l[3] == np.inf and np.all(np.isnan(l[4:7]))
    assert l[7] == math.log(5e-324)
