"""The tiled relaxation of rt_project_heights against the oracle where tiles
end (32 x 64 vertices), on domains the device classifies itself, and its
refusal of pairs that are not height functions of the domain."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

INF = np.iinfo(np.int32).max


def _case(model, sides):
    import randomtilings_b200 as rt
    from randomtilings_b200.project import extremal_heights

    code = rt.RT_DOMINO if model == "domino" else rt.RT_LOZENGE
    d = rt.DominoTiler.AztecDiamond(*sides) if model == "domino" else rt.LozengeTiler.Hexagon(*sides)
    return code, d, *extremal_heights(code, d)


# vertex sides around one tile row / column (n = 2 order + 6) and beyond two
@pytest.mark.parametrize("model,sides", [("domino", (1,)), ("domino", (13,)), ("domino", (14,)), ("domino", (29,)),
                                         ("domino", (30,)), ("domino", (62,)), ("lozenge", (1, 1, 1)),
                                         ("lozenge", (70, 9, 20)), ("lozenge", (5, 60, 61))])
def test_projection_over_tiles(model, sides):
    from randomtilings_b200.project import project_heights

    code, d, lo, hi = _case(model, sides)
    rng = np.random.default_rng(sum(sides))
    inside = lo != INF
    n = int(round(lo.size ** 0.5))
    ii, jj = np.divmod(np.arange(n * n), n)
    a, b = lo.astype(np.float64), hi.astype(np.float64)
    for t in ((a + b) / 2 + 30 * np.sin(ii / 9.0) * np.cos(jj / 31.0), a + (b - a) * rng.uniform(0, 1, n * n),
              np.where((ii // 32 + jj // 64) % 2 == 0, b, a), np.full(n * n, np.nan), np.full(n * n, np.inf)):
        t = np.where(inside, t, 0).astype(np.float32)
        got, st = project_heights(code, d, lo, hi, t)
        if np.isfinite(t).all():
            assert np.array_equal(got, po.project_heights(model, d, lo, hi, t))
            assert 0 <= st["lowered"] <= inside.sum() and 0 <= st["raised"] <= inside.sum()


@pytest.mark.parametrize("model,sides", [("domino", (20,)), ("lozenge", (9, 8, 7))])
def test_pairs_that_are_no_heights_are_refused(model, sides):
    import randomtilings_b200 as rt
    from randomtilings_b200.project import project_heights

    code, d, lo, hi = _case(model, sides)
    t = np.zeros(lo.size, dtype=np.float32)
    v = int(np.flatnonzero((lo != INF) & (hi > lo))[0])
    for at, value in ((lo, INF), (hi, INF), (hi, int(lo[v]) - 1), (hi, int(hi[v]) + 1)):
        keep = at[v]
        at[v] = value
        with pytest.raises(rt.RtError):
            project_heights(code, d, lo, hi, t)
        at[v] = keep
    with pytest.raises(rt.RtError):
        project_heights(code, d[:-1], lo, hi, t)
    project_heights(code, d, lo, hi, t)
