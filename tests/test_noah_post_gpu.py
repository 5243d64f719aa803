"""The post-step ranks a block's elements by the branches their columns take:
a column's results must not depend on its neighbours' columns.  Every other
element's groundwater changes between two runs (so that saturated, ice and
ice-free columns trade places in the blocks); the other elements come out with
the same bits, at element counts around a block's 128."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nelem", [127, 128, 129, 1201])
def test_a_columns_post_step_is_its_own(nelem):
    import torch

    import pihm_gpu.watershed as W
    from pihm_gpu import noah as N
    from pihm_gpu.capi import GpuRhs
    ws = W.generate(nelem, 10 if nelem < 500 else 100, seed=5)
    params, state = N.synthetic_noah(ws, seed=2)
    ne = ws.nelem
    y = W.reference_state(ws, 4)
    y2 = np.array(y, copy=True)
    moved = np.arange(ne) % 2 == 0
    depth = np.asarray(ws.arrays["depth"])
    y2[2 * ne:3 * ne][moved] = np.where(np.arange(ne) % 4 == 0, 2.0 * depth, 0.01 * depth)[moved]
    got = []
    for yy in (y, y2):
        g = GpuRhs(ws)
        g.noah_init(params, state)
        a, b = torch.from_numpy(y).cuda(), torch.from_numpy(yy).cuda()
        ai, bi, d = torch.empty_like(a), torch.empty_like(a), torch.empty_like(a)
        g.to_internal(a.data_ptr(), ai.data_ptr())
        g.to_internal(b.data_ptr(), bi.data_ptr())
        g.noah_begin(ai.data_ptr())
        g.noah_set_forcing(N.forcing(ws, 6, seed=3, diverse=True))
        g.noah_step(1800.0)
        g.rhs_device(ai.data_ptr(), d.data_ptr())
        for _ in range(2):
            g.noah_post_step(bi.data_ptr(), 60.0)
        got.append({f: g.noah_get(f) for f in ("smc", "sh2o", "smflxv", "runoff2_lyr", "infil", "runoff2", "fcr")})
    for f in got[0]:
        assert np.array_equal(got[0][f][~moved], got[1][f][~moved], equal_nan=True), f
    assert not np.array_equal(got[0]["smc"][moved], got[1]["smc"][moved])
