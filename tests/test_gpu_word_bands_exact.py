"""Bit-exact walks on bands with halos (rt_wordband.cu) against the oracle: halo
rows keep their own generators in step, runs of same-colour steps are phases, and
epochs reseed them; one CTA to many, bands of two rows and more, the last sizes
that fit, two lattices, weights."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _walk(tiler, t, steps, seed):
    a = np.array(t, dtype=np.int32)
    tiler.Walk(a, steps, seed)
    return a


@pytest.mark.parametrize("ctas", [0, 1, 2, 5, 9, 13, 24, 47])
def test_walks_match_the_oracle(monkeypatch, ctas):
    import randomtilings_b200 as rt

    if ctas:
        monkeypatch.setenv("RT_WALK_CTAS", str(ctas))
    t = rt.DominoTiler.MaxTiling(rt.DominoTiler.AztecDiamond(47))
    assert np.array_equal(_walk(rt.DominoTiler(), t, 251, 3), po.domino_walk(t, 251, 3))
    assert np.array_equal(_walk(rt.DominoTiler(kernel=1), t, 251, 4), po.domino_walk(t, 251, 4, cftp=True))
    t = rt.LozengeTiler.MinTiling(rt.LozengeTiler.Hexagon(40, 55, 31))
    assert np.array_equal(_walk(rt.LozengeTiler(), t, 251, 5), po.lozenge_walk(t, 251, 5))
    assert np.array_equal(_walk(rt.LozengeTiler(kernel=2), t, 251, 6), po.lozenge_walk(t, 251, 6, qweight=True))


@pytest.mark.parametrize("order", [2, 11, 12, 159, 160, 300, 420])
def test_edges_of_the_plan(order):
    """100 words on one CTA; word columns on both sides of 40; the largest bands."""
    import randomtilings_b200 as rt

    t = rt.DominoTiler.MinTiling(rt.DominoTiler.AztecDiamond(order))
    assert np.array_equal(_walk(rt.DominoTiler(), t, 60, 8), po.domino_walk(t, 60, 8))


@pytest.mark.parametrize("ctas", [1, 3, 6])
def test_two_lattices_and_epochs(monkeypatch, ctas):
    import randomtilings_b200 as rt

    monkeypatch.setenv("RT_WALK_CTAS", str(ctas))
    d = rt.DominoTiler.AztecDiamond(12)
    tmax, tmin = rt.DominoTiler.MaxTiling(d), rt.DominoTiler.MinTiling(d)
    got, st = rt.DominoTiler(kernel=1).CFTP(tmax, tmin, first_steps=16, master_seed=5, max_trials=20)
    want, trials, total, ok = po.cftp(tmax, tmin, 16, 5, max_trials=20)
    assert ok and st["coalesced"] and (st["trials"], st["total_steps"]) == (trials, total)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("ctas", [0, 4])
def test_weights(monkeypatch, ctas):
    import randomtilings_b200 as rt

    if ctas:
        monkeypatch.setenv("RT_WALK_CTAS", str(ctas))
    wh, wv = rt.DominoTiler.TwoPeriodicWeights(1.0, 0.6)
    t = rt.DominoTiler.MinTiling(rt.DominoTiler.AztecDiamond(33))
    tl = rt.DominoTiler(kernel=1)
    tl.SetWeights(wh, wv)
    assert np.array_equal(_walk(tl, t, 300, 21), po.domino_walk_weighted(t, [300], [21], wh, wv, single_walk=True))
