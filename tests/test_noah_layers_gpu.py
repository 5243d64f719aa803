"""Noah's kernels for columns of at most 4 layers against those for up to 11:
one column with a fifth layer sends the whole watershed through the second,
and every other column must come out with the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(ws, params, state, y, steps):
    import torch

    from pihm_gpu import noah as N
    from pihm_gpu.capi import GpuRhs
    g = GpuRhs(ws)
    g.noah_init(params, state)
    yr = torch.from_numpy(y).cuda()
    yi, yd = torch.empty_like(yr), torch.empty_like(yr)
    g.to_internal(yr.data_ptr(), yi.data_ptr())
    g.noah_begin(yi.data_ptr())
    out = []
    for k in range(steps):
        g.noah_set_forcing(N.forcing(ws, 6 + k, seed=3, diverse=True))
        g.noah_step(1800.0)
        g.rhs_device(yi.data_ptr(), yd.data_ptr())
        g.noah_post_step(yi.data_ptr(), 60.0)
        out.append({f: g.noah_get(f) for f in list(N.LAYER_FIELDS) + list(N.SCALAR_FIELDS)})
        out[-1]["ydot"] = yd.cpu().numpy()
    return out


@pytest.mark.parametrize("nelem", [60, 1201])
def test_four_layer_kernels_give_the_eleven_layer_kernels_bits(nelem):
    import pihm_gpu.watershed as W
    from pihm_gpu import noah as N
    ws = W.generate(nelem, 4 if nelem < 100 else 100, seed=5)
    params, state = N.synthetic_noah(ws, seed=2)
    y = W.reference_state(ws, 4)
    four = _run(ws, params, state, y, 3)
    p5 = {k: np.array(v, copy=True) for k, v in params.items()}
    s5 = {k: np.array(v, copy=True) for k, v in state.items()}
    e = ws.nelem // 2  # its last layer cut in two
    p5["nsoil"][e] = 5
    p5["sldpth"][e, 4] = 0.5 * p5["sldpth"][e, 3]
    p5["sldpth"][e, 3] -= p5["sldpth"][e, 4]
    for k in ("smc", "sh2o", "stc"):
        s5[k][e, 4] = s5[k][e, 3]
    eleven = _run(ws, p5, s5, y, 3)
    others = np.arange(ws.nelem) != e
    for a, b in zip(four, eleven):
        for f in N.LAYER_FIELDS:
            assert np.array_equal(a[f][others, :4], b[f][others, :4], equal_nan=True), f
        for f in N.SCALAR_FIELDS:
            assert np.array_equal(a[f][others], b[f][others], equal_nan=True), f
        assert np.all(np.isfinite(b["smc"][e, :5])) and np.all(np.isfinite(b["ydot"]))
