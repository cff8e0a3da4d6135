"""The six-vertex band kernel against the restatement: one CTA and many, halos of
four and two rows, rows of every length modulo the eight columns of a work item
and of several items a thread, thresholds that are all equal, that differ, and
that are 0 or 2^23, and two lattices."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

WEIGHTS = [None, (1.0, 2.0, 0.5, 1.5, 0.7, 1.1), (1e-20, 1.0, 1.0, 1.0, 1.0, 1e20), (1.0, 1.0, 1.0, 1.0, 3.0, 3.0)]


@pytest.mark.parametrize("n", [1, 2, 3, 15, 16, 17, 21, 30, 31, 63, 64, 90, 151, 333, 597])
@pytest.mark.parametrize("w", range(4))
def test_walks_match_the_restatement(n, w):
    import randomtilings_b200 as rt

    weights = WEIGHTS[w]
    t = rt.SixVertexTiler(weights=weights)
    h = np.array(rt.SixVertexTiler.MinHeights(n) if w % 2 else rt.SixVertexTiler.MaxHeights(n), dtype=np.int32)
    got = h.copy()
    t.Walk(got, 23, 2**40 + n, chain=w)
    want = po.sixv_walk(h, 23, 2**40 + n, chain=w, w=weights if weights else po.SIXV_UNIFORM)
    assert np.array_equal(got.reshape(-1), np.asarray(want).reshape(-1))


@pytest.mark.parametrize("n", [1300, 1601])
def test_wide_bands(n):
    """Bands of nine and eleven rows: halos of two rows, several items a thread."""
    import randomtilings_b200 as rt

    h = np.array(rt.SixVertexTiler.MaxHeights(n), dtype=np.int32)
    got = h.copy()
    rt.SixVertexTiler().Walk(got, 5, 3)
    assert np.array_equal(got.reshape(-1), np.asarray(po.sixv_walk(h, 5, 3)).reshape(-1))


@pytest.mark.parametrize("n,seed", [(20, 3), (50, 1)])
def test_two_lattices_with_unequal_thresholds(n, seed):
    import randomtilings_b200 as rt

    w = (1.0, 1.0, 1.0, 1.0, 1.2, 1.2)
    got, st = rt.SixVertexTiler(weights=w).CFTP(n, first_sweeps=16, master_seed=seed)
    want = po.sixv_cftp(n, 16, seed, w=w)
    assert np.array_equal(np.asarray(got).reshape(-1), np.asarray(want[0]).reshape(-1))
