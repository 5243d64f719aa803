"""A wait inside the one-launch evaluation that runs out (its limit set to no
look at the counter at all): the call reports an error and nothing else, and
the next evaluation starts afresh -- the separate kernels' bits, in a context
and in a batch arena, where the watersheds of that round alone fail."""
import ctypes

import numpy as np
import pytest

import pihm_gpu.watershed as W

pytestmark = pytest.mark.gpu

ERR_CUDA = -2


@pytest.mark.parametrize("nelem,nriver,surf", [(60, 4, 2), (5000, 390, 2), (5000, 390, 1)])
def test_context(nelem, nriver, surf):
    import torch

    from parity import apply, scenario
    from pihm_gpu.capi import GpuRhs
    ws = W.generate(nelem, nriver, seed=7)
    ws.surf_mode = surf
    ws, sc = scenario(ws, 2)
    a, b = GpuRhs(ws), GpuRhs(ws)
    b.set_profiling(True)  # the separate kernels
    for g in (a, b):
        apply(g, sc)
    limit = a.lib.pihm_gpu_set_wait_limit
    limit.argtypes = [ctypes.c_void_p, ctypes.c_int]
    y = np.asarray(sc["y"])
    d = torch.from_numpy(y).cuda()
    out = torch.empty_like(d)
    for call in range(3):
        assert limit(a.h, 0) == 0
        assert a.rhs_host(y)[1] == ERR_CUDA
        a.rhs_device(d.data_ptr(), out.data_ptr())
        assert a.status() == ERR_CUDA and a.status() == 0
        assert limit(a.h, -1) == 0
        (ga, ra), (gb, rb) = a.rhs_host(y * (1.0 + 0.01 * call)), b.rhs_host(y * (1.0 + 0.01 * call))
        assert (ra, rb) == (0, 0) and np.array_equal(ga, gb), call


def test_batch():
    from pihm_gpu.batch import DONE, FAILED, Batch, limits_for
    from test_batch_gpu import _alone, _case, _same
    cases = [_case(300, 71, 1), _case(1000, 72, 1)]
    want = [_alone(c) for c in cases]
    b = Batch(limits_for([c["ws"] for c in cases], 2))
    limit = b.lib.pihm_batch_set_wait_limit
    limit.argtypes = [ctypes.c_void_p, ctypes.c_int]
    try:
        for _ in range(2):
            assert limit(b.h, 0) == 0
            ids = b.add_many(cases)
            b.step()
            for i in ids:
                assert b.poll(i)[0] == FAILED
                b.release(i)
            assert limit(b.h, -1) == 0
            ids = b.add_many(cases)
            b.step()
            for k, i in enumerate(ids):
                assert b.poll(i) == (DONE, 0)
                _same(b.result(i), want[k], str(k))
                b.release(i)
    finally:
        b.close()
