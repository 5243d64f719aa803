"""The program kernel's layouts (a warp of the reduction order per block, or
whole blocks with 1, 2 or 4 entries a thread): every one gives a watershed the
single-watershed path's bits, at the sizes where the choice changes -- a
watershed of one block, at 76 and 77 blocks of the reduction order, and rounds
below and above 400 blocks."""
import pytest

from pihm_gpu.batch import Batch, limits_for
from test_batch_gpu import _alone, _case, _same

pytestmark = pytest.mark.gpu


def _blocks(ws):
    return -(-ws.neq // 1024)


@pytest.mark.parametrize("sizes,variant", [([60, 1000], -1), ([24_300, 60], -1), ([25_900, 60], -1),
                                           ([20_000] * 7, -1), ([24_300, 1000], 0), ([24_300, 1000], 2)])
def test_program_layouts_same_trajectory(sizes, variant):
    made = {n: _case(n, 40 + i, 1) for i, n in enumerate(dict.fromkeys(sizes))}
    cases = [made[n] for n in sizes]
    if sizes[0] == 24_300:
        assert _blocks(cases[0]["ws"]) <= 76
    if sizes[0] == 25_900:
        assert _blocks(cases[0]["ws"]) > 76
    if len(sizes) > 2:
        assert sum(_blocks(c["ws"]) for c in cases) > 400
    want = {n: _alone(c) for n, c in made.items()}
    b = Batch(limits_for([c["ws"] for c in cases], 4))
    try:
        if variant >= 0:
            b.set_program_variant(variant)
        ids = b.add_many(cases)
        assert None not in ids
        b.step()
        for n, i in zip(sizes, ids):
            _same(b.result(i), want[n], f"{n} elements")
    finally:
        b.close()


def test_uploads_beside_each_other_and_with_boundary_values():
    """Watersheds admitted together (one upload that moves every index to its
    watershed's ranges), the middle one with element and river boundary
    values, and one admitted into a released watershed's ranges."""
    from backends import GpuBackend
    from parity import scenario
    from pihm_gpu.solver import run_steps
    cases = [_case(700, 51, 1), _case(1500, 52, 1), _case(300, 53, 1)]
    ws, sc = scenario(cases[1]["ws"], 3, bc=True)
    cases[1].update(ws=ws, elem_bc=sc["elem_bc"], river_bc=sc["river_bc"])
    want = []
    for c in cases:
        g = GpuBackend(c["ws"], c["y0"], c["pcp"], c["edir"], c["ett"])
        try:
            if "elem_bc" in c:
                g.g.set_bc(c["elem_bc"], c["river_bc"])
            r = run_steps(g, c["ctrl"], 1, g.set_forcing, record_every=1, outlet=c["outlet"])
        finally:
            g.close()
        want.append(dict(y=r["states"][-1], outlet=r["outlet"], stats=r["stats"]))
    b = Batch(limits_for([c["ws"] for c in cases], 4))
    try:
        ids = b.add_many(cases)
        b.step()
        for k, i in enumerate(ids):
            _same(b.result(i), want[k], f"case {k}")
        b.release(ids[1])
        again = b.add_many([cases[1]])
        b.step()
        _same(b.result(again[0]), want[1], "readmitted")
    finally:
        b.close()
