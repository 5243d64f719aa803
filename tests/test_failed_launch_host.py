"""A kernel launch that fails is reported by the call that made it and leaves
nothing behind for the next one, which succeeds (on the CPU, over the stand-in
for the CUDA runtime in fake_cudart.cpp): the evaluation in one launch and in
several, the reorderings, the land-surface step."""
import pytest

from test_nv_queue_host import _child, fake  # noqa: F401


@pytest.mark.parametrize("nelem", [60, 16_000])
def test_the_next_call_succeeds(fake, nelem):  # noqa: F811
    _child(fake, f"""
import pihm_gpu.land as L
from pihm_gpu.capi import GpuRhs, PihmGpuError
fake.fake_launches.restype = ctypes.c_long
ws = W.generate({nelem}, {nelem} // 15, seed=1)
g = GpuRhs(ws)
land = L.synthetic_land(ws, seed=1, hours=6)
g.land_init(land)
time = L.epoch("2009-01-01 03:00")
y, d = np.zeros(ws.neq), np.zeros(ws.neq)
host = lambda: g.rhs_host(y)[1]
calls = dict(rhs=lambda: g.rhs_device(y.ctypes.data, d.ctypes.data),
             reorder=lambda: g.to_reference(y.ctypes.data, d.ctypes.data),
             back=lambda: g.to_internal(y.ctypes.data, d.ctypes.data),
             land=lambda: g.land_step(time, 900.0, y.ctypes.data))
for name, call in calls.items():
    call()  # (a month's table on the first step)
    fake.fake_reset()
    call()
    n = fake.fake_launches()
    assert (n >= 4 if name == "rhs" and ws.nelem == 16_000 else n >= 1), (name, n)
    for k in range(n):
        fake.fake_reset()
        fake.fake_refuse_any(k)
        try:
            call()
            raise AssertionError((name, k))
        except PihmGpuError as e:
            assert e.rc == -2, (name, k)
        fake.fake_refuse_any(-1)
        assert g.status() == 0, (name, k)
        call()
""")
