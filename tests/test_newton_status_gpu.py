"""A right-hand side that turns NaN in a Newton iteration, with its status
read back at once (deferred scalars off) and with the next norm: the same
return, counters and state, and the integrator usable afterwards."""
import ctypes

import numpy as np
import pytest

import pihm_gpu.solver as S
import pihm_gpu.watershed as W
import pihm_gpu.workloads as WL
from backends import GpuBackend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nelem", [300, 60_000])
def test_nan_in_newton_evaluation(nelem):
    ws = W.generate(nelem, WL.river_count(nelem), seed=5)
    pcp, edir, ett = WL.step_forcing(ws, 3, 60.0, seed=3)
    out = {}
    for mode in (0, -1):
        b = GpuBackend(ws, W.relax_state(ws), pcp, edir, ett)
        bdf = S.Bdf()
        try:
            lib = bdf.lib
            ctrl = S.StepControl()
            assert lib.pihm_bdf_init(bdf.h, b.rhs, 0.0, b.y) == 0
            assert lib.pihm_bdf_ss_tolerances(bdf.h, ctrl.reltol, ctrl.abstol) == 0
            assert lib.pihm_bdf_set_user_data(bdf.h, b.user_data) == 0
            assert lib.pihm_bdf_set_init_step(bdf.h, ctrl.initstep) == 0
            assert lib.pihm_bdf_set_deferred_scalars(bdf.h, mode) == 0
            t, rcs, states = ctypes.c_double(0.0), [], []
            for k, bad in ((0, False), (1, True), (2, False)):
                b.set_forcing(k)
                if bad:
                    b.g.set_forcing(np.full(ws.nelem, np.nan), np.zeros(ws.nelem), np.zeros(ws.nelem))
                rcs.append(lib.pihm_bdf_solve(bdf.h, 60.0 * (k + 1), b.y, ctypes.byref(t)))
                states.append(b.read_state())
            s = bdf.stats()
            out[mode] = (rcs, states, [getattr(s, n) for n, _ in s._fields_])
        finally:
            bdf.close()
            b.close()
    assert out[0][0][0] == 0 and out[0][0][1] < 0
    assert out[-1][0] == out[0][0] and out[-1][2] == out[0][2]
    for a, c in zip(out[-1][1], out[0][1]):
        assert np.array_equal(a, c)
