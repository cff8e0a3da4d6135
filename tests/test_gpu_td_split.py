"""The triangle-dimer arrays set up on the device (td_split_kernel): states of
covers and of arbitrary values, the smallest sides, and what is refused."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 10, 30, 66, 70])
@pytest.mark.parametrize("high", [2**4, 2**6, 2**31])
def test_arbitrary_values(n, high):
    """Every array enters a move's outcome within a few steps."""
    import randomtilings_b200 as rt

    lo = -high if high == 2**31 else 0
    t = np.random.default_rng(n).integers(lo, high, n * n).astype(np.int32)
    a = t.copy()
    rt.TriangleDimerTiler().Walk(a, 40, 3)
    assert np.array_equal(a, po.tridimer_walk(t, 40, 3))


def test_batches_refuse_what_is_no_cover():
    import randomtilings_b200 as rt

    good = np.array(rt.TriangleDimerTiler.BiboneHexagon(9), dtype=np.int32)
    n = int(round(len(good) ** 0.5))
    for value in (16, -1):
        t = good.copy()
        t[n + 1] = value
        b = rt.Batch()
        b.add(rt.RT_TRIDIMER, t, 1)
        with pytest.raises(rt.RtError, match="out of range"):
            b.run(1)
        b.close()
