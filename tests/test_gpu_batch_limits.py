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
