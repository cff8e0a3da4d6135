"""The triangle-dimer walk on bit planes (rt_td.cu) against the oracle: one CTA
to the largest cluster, bands of four rows and of uneven heights, one and two
words of columns, states carried from one run to the next, a table of generator
parameters, and starts that are no dimer covers."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _walk(tiler, t, steps, seed):
    a = np.array(t, dtype=np.int32)
    tiler.Walk(a, steps, seed)
    return a


# array sides 8 (cluster of 8 rows), 22, 62 and 66 (one, two, three words)
@pytest.mark.parametrize("side", [2, 9, 29, 31])
@pytest.mark.parametrize("ctas", [0, 1, 2, 5, 16])
def test_walks_match_the_oracle(monkeypatch, side, ctas):
    import randomtilings_b200 as rt

    if ctas:
        monkeypatch.setenv("RT_WALK_CTAS", str(ctas))
    t = rt.TriangleDimerTiler.BiboneHexagon(side)
    assert np.array_equal(_walk(rt.TriangleDimerTiler(), t, 150, 9), po.tridimer_walk(t, 150, 9))
    got = _walk(rt.TriangleDimerTiler(rng=rt.RT_RNG_PHILOX), t, 150, 2**40 + 1)
    assert np.array_equal(got, po.walk_fast("tridimer", t, 150, 2**40 + 1))


def test_runs_continue():
    """A run leaves every array as the reference does, wherever it stops."""
    import randomtilings_b200 as rt

    t = rt.TriangleDimerTiler.BiboneHexagon(12)
    want = np.array(t, dtype=np.int32)
    tl = rt.TriangleDimerTiler()
    tl.upload(t)
    out = np.zeros(len(t), dtype=np.int32)
    for k, steps in enumerate((1, 2, 3, 5, 40, 1, 60)):
        tl.run(steps, 70 + k)
        want = po.tridimer_walk(want, steps, 70 + k)
        tl.download(out)
        assert np.array_equal(out, want), (k, steps)


def test_parameter_table():
    import randomtilings_b200 as rt

    t = rt.TriangleDimerTiler.BiboneHexagon(10)
    m = int(round(len(t) ** 0.5)) // 2
    table = np.random.default_rng(3).integers(0, 2**32, (m * m, 3), dtype=np.uint32)
    tl = rt.TriangleDimerTiler()
    tl.SetTinyMTTable(table)
    assert np.array_equal(_walk(tl, t, 200, 4), po.tridimer_walk(t, 200, 4, params=table))


@pytest.mark.parametrize("high", [16, 300])
def test_starts_that_are_no_covers(monkeypatch, high):
    """Both kernels give the same tiling: values that fit the planes stay exact,
    others take the int32 kernel."""
    import randomtilings_b200 as rt

    t = np.random.default_rng(high).integers(0, high, 40 * 40).astype(np.int32)
    got = _walk(rt.TriangleDimerTiler(), t, 120, 6)
    monkeypatch.setenv("RT_WALK_KERNEL", "generic")
    assert np.array_equal(got, _walk(rt.TriangleDimerTiler(), t, 120, 6))
