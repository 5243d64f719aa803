"""The most watersheds one round of the batch takes: the program kernel stages
every watershed's first block (4 bytes) beside a program of 1,920 bytes and its
reductions' 272 in 48 KB of shared memory.  11,660 watersheds of one element
each follow the trajectory of one alone."""
import numpy as np
import pytest

import pihm_gpu.watershed as W

pytestmark = pytest.mark.gpu

SYSTEMS = 11_660


def test_every_watershed_of_a_full_round():
    from pihm_gpu.batch import Batch, limits_for
    from test_batch_gpu import _case
    from test_rhs_edgeless_gpu import _alone, _edgeless
    ws = _edgeless("one element")
    c = dict(_case(60, 81, 2), ws=ws, y0=W.reference_state(ws, seed=3), outlet=-1)
    c["pcp"], c["edir"], c["ett"] = (np.array(c[k][:2]) for k in ("pcp", "edir", "ett"))
    want, stats = _alone(c)
    b = Batch(limits_for([ws] * SYSTEMS, 2))
    try:
        ids = b.add_many([c] * SYSTEMS)
        assert None not in ids
        assert b.step() == 0
        for i in ids:
            got = b.result(i)
            assert np.array_equal(got["y"], want) and got["stats"].nst == stats.nst
    finally:
        b.close()
