"""The bit-plane walk with one word per thread (rt_planeband.cu) against the
oracle: one, two and four rows a thread, one CTA to the whole GPU, uneven bands,
halo depths that are and are not a multiple of the four steps drawn at once or
of the colour round, and two lattices."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _tiler(rt, monkeypatch, model, kernel, ctas, depth, **kw):
    monkeypatch.setenv("RT_WALK_CTAS", str(ctas))
    monkeypatch.setenv("RT_PLANE_DEPTH", str(depth))
    cls = rt.DominoTiler if model == "domino" else rt.LozengeTiler
    return cls(kernel=kernel, rng=rt.RT_RNG_PLANES, **kw)


# Dominoes of order 130: 264 rows of 5 words (8 with padding); hexagons of side
# 90: 189 rows of 2 words (4).  With one CTA the block holds them at four / two
# rows a thread, with more at two and one.
@pytest.mark.parametrize("model,kernel", [("domino", 0), ("domino", 1), ("lozenge", 0)])
@pytest.mark.parametrize("ctas,depth", [(0, 0), (1, 0), (2, 0), (3, 11), (4, 5), (12, 9), (12, 0), (100, 0)])
def test_walks_match_the_oracle(monkeypatch, model, kernel, ctas, depth):
    import randomtilings_b200 as rt

    D, L = rt.DominoTiler, rt.LozengeTiler
    t = D.MinTiling(D.AztecDiamond(130)) if model == "domino" else L.MinTiling(L.Hexagon(90, 90, 90))
    tl = _tiler(rt, monkeypatch, model, kernel, ctas, depth, chain=2)
    got = np.array(t, dtype=np.int32)
    tl.Walk(got, 75, 2**35 + 3)
    assert np.array_equal(got, po.walk_planes("domino_cftp" if kernel else model, t, 75, 2**35 + 3, chain=2))


@pytest.mark.parametrize("model,kernel", [("domino", 1), ("lozenge", 0)])
@pytest.mark.parametrize("ctas", [1, 2, 6])
def test_two_lattices(monkeypatch, model, kernel, ctas):
    """Two starts three steps apart meet after a few short epochs."""
    import randomtilings_b200 as rt

    D, L = rt.DominoTiler, rt.LozengeTiler
    t = D.MinTiling(D.AztecDiamond(130)) if model == "domino" else L.MinTiling(L.Hexagon(90, 90, 90))
    name = "domino_cftp" if kernel else model
    u = po.walk_planes(name, t, 3, 5)
    tl = _tiler(rt, monkeypatch, model, kernel, ctas, 0)
    got, st = tl.CFTP(u, t, first_steps=8, master_seed=9, max_trials=4)
    want, trials, total, ok = po.cftp(u, t, 8, 9, max_trials=4, model=name, planes=True)
    assert (st["coalesced"], st["trials"], st["total_steps"]) == (ok, trials, total)
    assert np.array_equal(got, want)
