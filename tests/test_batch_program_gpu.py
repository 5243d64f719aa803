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
