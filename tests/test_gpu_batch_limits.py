"""The largest chains that a batch holds, at each cluster size: a band fills
shared memory, and the kernels leave out what they can do without."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _batch(rt, model, t, key, sweeps, cluster, block=512):
    b = rt.Batch()
    b.add(model, t, key, chain=3)
    b.set_tuning(False, cluster, block)
    b.run(sweeps)
    out, info = b.download(0), b.info()
    b.close()
    (plan,) = info["plans"].values()
    return out, plan["cluster"]


@pytest.mark.parametrize("side", [945, 947])
def test_lozenge_chains_that_leave_no_room_for_tables(side):
    """Sides 1,899 and 1,902: 36 bytes of a CTA's shared memory are left."""
    import randomtilings_b200 as rt

    t = rt.LozengeTiler.MinTiling(rt.LozengeTiler.Hexagon(side, side, side))
    got, cluster = _batch(rt, rt.RT_LOZENGE, t, 2**41 + 7, 3, 16)
    assert cluster == 16
    assert np.array_equal(got, po.walk_fast("lozenge", t, 9, 2**41 + 7, chain=3))


# (hexagon side, cluster): arrays of side 2 s + 8.  A cluster of 2 holds sides of
# 210 with the deepest halo, 226 with one row, 248 with a dimer cover's planes;
# of 8: 400, 480 and 512; of 16: 528, 688 and 720.
@pytest.mark.parametrize("side,cluster", [(101, 2), (102, 2), (109, 2), (110, 2), (120, 2), (196, 8), (200, 8), (236, 8),
                                          (237, 8), (252, 8), (260, 16), (340, 16), (341, 16), (356, 16)])
def test_triangle_dimer_chains(side, cluster):
    import randomtilings_b200 as rt

    t = np.asarray(rt.TriangleDimerTiler.BiboneHexagon(side), dtype=np.int32)
    got, used = _batch(rt, rt.RT_TRIDIMER, t, 2**41 + 7, 2, cluster)
    assert used == cluster
    assert np.array_equal(got, po.walk_fast("tridimer", t, 60, 2**41 + 7, chain=3))


def test_the_tuner_holds_the_largest_triangle_dimer_chain():
    import randomtilings_b200 as rt

    t = np.asarray(rt.TriangleDimerTiler.BiboneHexagon(252), dtype=np.int32)
    small = np.asarray(rt.TriangleDimerTiler.BiboneHexagon(9), dtype=np.int32)
    b = rt.Batch()
    for c, x in enumerate((t, small)):
        b.add(rt.RT_TRIDIMER, x, 5 + c, chain=c)
    b.run(1)
    for c, x in enumerate((t, small)):
        assert np.array_equal(b.download(c), po.walk_fast("tridimer", x, 30, 5 + c, chain=c))
    b.close()
