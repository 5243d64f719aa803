"""Meshes without interior edges under the diffusion wave: one element, two
elements on either side of a segment, elements that touch only segments and
the boundary (more than one block of each kind).  The one-launch evaluation's
barriers then have no edge blocks to hold the elements.  The same bits as the
separate kernels on the device and the host entry points, the oracle's rows,
and in a batch arena that holds such a watershed alone and then one with
edges."""
import numpy as np
import pytest

import pihm_gpu.watershed as W

pytestmark = pytest.mark.gpu


def _cut(nelem, nriver, elems, segs):
    """The elements and segments of a generated mesh by themselves, every
    interior edge a boundary and every segment an outlet."""
    ws = W.generate(nelem, nriver, seed=nelem)
    elems, segs = np.asarray(elems), np.asarray(segs, int)
    new_e = np.zeros(nelem + 1, np.int32)
    new_e[elems + 1] = np.arange(1, elems.size + 1)
    new_s = np.zeros(nriver + 1, np.int32)
    new_s[segs + 1] = np.arange(1, segs.size + 1)
    a = {}
    for k in W.ELEM_INT_FIELDS + W.ELEM_F64_FIELDS:
        v = ws.arrays[k]
        a[k] = (v.reshape(nelem, 3)[elems].reshape(-1) if k in W.PER_EDGE else v[elems]).copy()
    for k in W.RIVER_INT_FIELDS + W.RIVER_F64_FIELDS:
        a[k] = ws.arrays[k][segs].copy()
    a["nabr"] = np.where(a["nabr"] < 0, -new_s[np.maximum(-a["nabr"], 0)], 0).astype(np.int32)
    a["bc_type"] = np.zeros_like(a["bc_type"])
    a["down"] = np.full(segs.size, W.CRIT_DPTH, np.int32)
    a["leftele"], a["rightele"] = new_e[a["leftele"]], new_e[a["rightele"]]
    return W.Watershed(int(elems.size), int(segs.size), a)


def _edgeless(name):
    if name == "one element":
        return _cut(60, 4, [17], [])
    ws = W.generate(60, 4, seed=60)
    if name == "two and a segment":
        return _cut(60, 4, [ws.arrays["leftele"][1] - 1, ws.arrays["rightele"][1] - 1], [1])
    return _cut(3000, 240, np.arange(3000), np.arange(240))


NAMES = ["one element", "two and a segment", "3,000 apart"]


def _rhs(ws, sc, separate):
    from parity import apply
    from pihm_gpu.capi import GpuRhs
    g = GpuRhs(ws)
    apply(g, sc)
    g.set_diagnostics(True)
    g.set_profiling(separate)
    return g


@pytest.mark.parametrize("name", NAMES)
def test_evaluation(name):
    import torch

    from oracle import Oracle
    from parity import apply, compare, row_scales, scenario
    ws, sc = scenario(_edgeless(name), 4)
    a, b, o = _rhs(ws, sc, False), _rhs(ws, sc, True), Oracle(ws)
    apply(o, sc)
    yr = torch.empty(ws.neq, dtype=torch.float64, device="cuda")
    yi, da, db = torch.empty_like(yr), torch.empty_like(yr), torch.empty_like(yr)
    for call in range(20):
        y = np.asarray(sc["y"]) * (1.0 + 0.01 * call)
        (ga, ra), (gb, rb), (want, ro) = a.rhs_host(y), b.rhs_host(y), o.rhs(y)
        assert (ra, rb, ro) == (0, 0, 0) and np.array_equal(ga, gb)
        ok, worst, row = compare(ga, want, row_scales(ws, o.fluxes(), sc["pcpdrp"], sc["edir"], sc["ett"]))
        assert ok, (worst, row)
        yr.copy_(torch.from_numpy(y))
        for g, d in ((a, da), (b, db)):
            torch.cuda.synchronize()
            g.to_internal(yr.data_ptr(), yi.data_ptr())
            g.rhs_device(yi.data_ptr(), d.data_ptr())
            assert g.status() == 0
        assert torch.equal(da, db)
        o.rhs(y)  # the river banks' carried flux: as many evaluations as the contexts made


def _alone(c):
    from backends import GpuBackend
    from pihm_gpu.solver import run_steps
    b = GpuBackend(c["ws"], c["y0"], c["pcp"], c["edir"], c["ett"])
    try:
        r = run_steps(b, c["ctrl"], 2, b.set_forcing, record_every=2)
    finally:
        b.close()
    return r["states"][-1], r["stats"]


def test_arena_with_and_without_edges():
    from pihm_gpu.batch import Batch, limits_for
    from test_batch_gpu import _case
    cases = [_case(1000, 61, 2)]
    for k, name in enumerate(NAMES):
        ws = _edgeless(name)
        cases.append(dict(_case(60, 62 + k, 2), ws=ws, y0=W.reference_state(ws, seed=k)))
    for c in cases:
        c["outlet"] = -1
    want = [_alone(c) for c in cases]
    b = Batch(limits_for([c["ws"] for c in cases], 8))
    try:
        for group in ([1], [2], [0], [3], [1, 2], [0, 1, 2, 3]):
            ids = b.add_many([cases[k] for k in group])
            assert None not in ids
            b.step()
            for k, i in zip(group, ids):
                got = b.result(i)
                assert np.array_equal(got["y"], want[k][0]), (group, k)
                assert (got["stats"].nst, got["stats"].nfe) == (want[k][1].nst, want[k][1].nfe)
                b.release(i)
    finally:
        b.close()
