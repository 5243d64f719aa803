"""The one-launch evaluation of small meshes (k_rhs_fused) against the
separate kernels, which a context with per-kernel timing on keeps using: the
same bits for every row and flux, over consecutive calls (the river banks'
carried flux), through the device and the host entry points, under boundary
conditions, in Flux-PIHM mode, and replayed from a CUDA graph.  The sizes
stand at the edges of the launch rule: fewer items than a block, one item a
thread at 128 registers, at 64, and sizes past the last that fits (155,648
items: elements twice, interior edges, four parts of every segment)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FLUXES = ("ovlflow", "subsurf", "infil", "rechg", "et_split", "rivflow")


def _context(ws, sc, separate):
    from parity import apply
    from pihm_gpu.capi import GpuRhs
    g = GpuRhs(ws)
    apply(g, sc)
    g.set_diagnostics(True)
    g.set_profiling(separate)
    return g


@pytest.mark.parametrize("nelem,nriver,mesh,surf,riv,bc,noah", [
    (60, 4, "grid", 2, 2, False, False),
    (1000, 100, "grid", 2, 2, True, False),
    (1000, 100, "grid", 1, 1, False, True),
    (4999, 390, "scattered", 1, 2, True, False),
    (19000, 1100, "grid", 2, 2, False, True),
    (23000, 1300, "scattered", 2, 2, True, False),
    (41000, 2200, "grid", 2, 1, True, False),
    (43000, 2200, "grid", 2, 1, False, False),
    (48000, 2400, "grid", 2, 2, False, False),
])
def test_one_launch_gives_the_separate_kernels_bits(nelem, nriver, mesh, surf, riv, bc, noah):
    import pihm_gpu.watershed as W
    from parity import scenario
    ws = W.generate(nelem, nriver, seed=nelem, mesh=mesh)
    ws.surf_mode, ws.riv_mode = surf, riv
    ws, sc = scenario(ws, 5, bc=bc, noah=noah)
    a, b = _context(ws, sc, False), _context(ws, sc, True)
    for call in range(3):
        y = np.asarray(sc["y"]) * (1.0 + 0.01 * call)
        n0 = a.launch_count()
        (ya, ra), (yb, rb) = a.rhs_host(y), b.rhs_host(y)
        assert ra == 0 and rb == 0
        if nelem <= 41000:
            assert a.launch_count() - n0 == 2  # the evaluation and the reordering
        assert np.array_equal(ya, yb)
        fa, fb = a.fluxes(), b.fluxes()
        for k in FLUXES:
            assert np.array_equal(fa[k], fb[k]), (k, call)


def test_one_launch_on_device_vectors_and_from_a_graph():
    import torch

    import pihm_gpu.watershed as W
    from parity import scenario
    ws, sc = scenario(W.generate(3000, 240, seed=9), 3)
    a, b = _context(ws, sc, False), _context(ws, sc, True)
    yr = torch.from_numpy(np.asarray(sc["y"], np.float64)).cuda()
    y, da, db = torch.empty_like(yr), torch.empty_like(yr), torch.empty_like(yr)
    a.to_internal(yr.data_ptr(), y.data_ptr())
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    a.set_stream(s.cuda_stream)
    with torch.cuda.stream(s):
        a.rhs_device(y.data_ptr(), da.data_ptr())
    s.synchronize()
    b.rhs_device(y.data_ptr(), db.data_ptr())
    torch.cuda.synchronize()
    assert torch.equal(da, db)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        a.rhs_device(y.data_ptr(), da.data_ptr())
    for k in range(3):  # each replay sees the flux the one before it carried
        y.mul_(1.0 + 0.02 * k)
        da.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        b.rhs_device(y.data_ptr(), db.data_ptr())
        torch.cuda.synchronize()
        assert torch.equal(da, db), k
    assert a.status() == 0


def test_a_nan_state_is_reported():
    import pihm_gpu.watershed as W
    from parity import scenario
    ws, sc = scenario(W.generate(1000, 100, seed=2), 1)
    a = _context(ws, sc, False)
    y = np.asarray(sc["y"]).copy()
    y[ws.nelem + 17] = np.nan  # unsaturated storage: the powers leave their ranges
    _, rc = a.rhs_host(y)
    b = _context(ws, sc, True)
    _, rc2 = b.rhs_host(y)
    assert rc == rc2
    got, rc = a.rhs_host(np.asarray(sc["y"]))  # and the next evaluation is a valid one
    assert rc == 0 and np.all(np.isfinite(got))
