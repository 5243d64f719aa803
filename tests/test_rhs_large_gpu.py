"""Large meshes' five dependent launches, whose blocks start while the kernel
before them ends, against the separate, serialised kernels of a context with
per-kernel timing: the same bits for evaluations queued back to back without
a synchronisation, alternating between states, on device vectors (also
replayed from a CUDA graph) and from the host; with and without the gradient
kernel, and with a single river segment."""
import numpy as np
import pytest

from test_rhs_fused_gpu import _context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nelem,nriver,mesh,surf,bc,noah", [
    (60_000, 2600, "grid", 2, True, False),
    (50_001, 2100, "scattered", 1, False, True),
    (90_000, 4, "grid", 2, False, False),
])
def test_dependent_launches_give_the_serialised_bits(nelem, nriver, mesh, surf, bc, noah):
    import torch

    import pihm_gpu.watershed as W
    from parity import scenario
    ws = W.generate(nelem, nriver, seed=nelem, mesh=mesh)
    ws.surf_mode = surf
    ws, sc = scenario(ws, 5, bc=bc, noah=noah)
    a, b = _context(ws, sc, False), _context(ws, sc, True)
    base = np.asarray(sc["y"], np.float64)
    y = []
    for k in range(3):
        yr = torch.from_numpy(base * (1.0 + 0.05 * k)).cuda()
        yi = torch.empty_like(yr)
        a.to_internal(yr.data_ptr(), yi.data_ptr())
        torch.cuda.synchronize()
        y.append(yi)
    s = torch.cuda.Stream()
    a.set_stream(s.cuda_stream)
    n = 24
    da, db = [torch.empty_like(y[0]) for _ in range(n)], torch.empty_like(y[0])
    torch.cuda.synchronize()
    for k in range(n):
        a.rhs_device(y[k % 3].data_ptr(), da[k].data_ptr())
    s.synchronize()
    want = []
    for k in range(n):
        b.rhs_device(y[k % 3].data_ptr(), db.data_ptr())
        torch.cuda.synchronize()
        want.append(db.clone())
        assert torch.equal(da[k], want[k]), k
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        for k in range(3):
            a.rhs_device(y[k].data_ptr(), da[k].data_ptr())
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    for k in range(3):  # as the last rounds above: the carried flux has gone round too
        assert torch.equal(da[k], want[n - 3 + k]), k
    a.set_stream(0)
    for k in range(4):
        (ya, ra), (yb, rb) = a.rhs_host(base * (1.0 + 0.05 * (k % 2))), b.rhs_host(base * (1.0 + 0.05 * (k % 2)))
        assert ra == 0 and rb == 0
        if k > 0:  # the first sees each context's own last device evaluation
            assert np.array_equal(ya, yb), k
    assert a.status() == 0 and b.status() == 0
