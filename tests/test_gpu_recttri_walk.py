"""The rectangle-triangle walk with one site per thread (rt_recttri.cu) against
the oracle: one CTA, clusters and whole-GPU grids, bands of one row, uneven
bands and blocks on both sides of the register bound, runs of more draws than
are made ahead, a parameter table, non-unit weights, any starting values, and
the generic kernel beyond the bands that fit."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

W = np.array([0.0, 1.0, 2.0, 0.5, 1.5, 0.7, 1.1, 1.5, 0.7, 1.1, 0.3, 3.0, 1.0, 0.3, 3.0, 1.0], dtype=np.float32)


def _walk(tiler, t, steps, seed):
    a = np.array(t, dtype=np.int32)
    tiler.Walk(a, steps, seed)
    return a


def _both_modes(t, steps, **kw):
    import randomtilings_b200 as rt

    w = kw.get("weights")
    assert np.array_equal(_walk(rt.RectTriangleTiler(**kw), t, steps, 9), po.recttri_walk(t, steps, 9, weights=w))
    got = _walk(rt.RectTriangleTiler(rng=rt.RT_RNG_PHILOX, **kw), t, steps, 2**40 + 1)
    assert np.array_equal(got, po.walk_fast("recttri", t, steps, 2**40 + 1, weights=w))


@pytest.mark.parametrize("side", [1, 6, 20, 37])
@pytest.mark.parametrize("ctas", [0, 1, 2, 7, 16, 40])
def test_walks_match_the_oracle(monkeypatch, side, ctas):
    import randomtilings_b200 as rt

    if ctas:
        monkeypatch.setenv("RT_WALK_CTAS", str(ctas))
    _both_modes(rt.RectTriangleTiler.maxHex(side), 400)


@pytest.mark.parametrize("side", [64, 90, 200])
def test_large(side):
    """One cluster, the largest blocks of one, and the whole GPU."""
    import randomtilings_b200 as rt

    _both_modes(rt.RectTriangleTiler.maxHex(side), 60, weights=W)


@pytest.mark.parametrize("side", [12, 40])
def test_any_values_and_parameter_table(monkeypatch, side):
    import randomtilings_b200 as rt

    n = int(round(len(rt.RectTriangleTiler.maxHex(side)) ** 0.5))
    rng = np.random.default_rng(side)
    t = rng.integers(-(2**31), 2**31, n * n).astype(np.int32)
    _both_modes(t, 200)
    table = rng.integers(0, 2**32, (n * n // 3, 3), dtype=np.uint64).astype(np.uint32)
    s = rt.RectTriangleTiler.maxHex(side)
    for kernel in ("auto", "generic"):
        monkeypatch.setenv("RT_WALK_KERNEL", kernel)
        tl = rt.RectTriangleTiler(weights=W)
        tl.SetTinyMTTable(table)
        assert np.array_equal(_walk(tl, s, 300, 4), po.recttri_walk(s, 300, 4, weights=W, params=table))


@pytest.mark.parametrize("n", [237, 240])
def test_batches_with_and_without_the_table(n):
    """Alone on one CTA a side of 240 fills shared memory: no room for the table of moves."""
    import randomtilings_b200 as rt

    t = np.resize(rt.RectTriangleTiler.maxHex(20), n * n).astype(np.int32)
    b = rt.Batch()
    b.add(rt.RT_RECTTRI, t, 77, chain=0)
    b.set_tuning(False, 1, 512)
    b.run(10)
    got = b.download(0)
    b.close()
    assert np.array_equal(got, po.walk_fast("recttri", t, 30, 77))
