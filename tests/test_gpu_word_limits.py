"""The last sides that the fast mode's word kernel holds: a band fills shared
memory to within 200 bytes."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,size", [("domino", 2822), ("domino", 2829), ("domino_cftp", 2829), ("lozenge", 2828),
                                        ("qlozenge", 2828)])
def test_largest_sides(monkeypatch, model, size):
    import randomtilings_b200 as rt

    monkeypatch.setenv("RT_WALK_KERNEL", "word")
    if model.startswith("domino"):
        t = rt.DominoTiler.MinTiling(rt.DominoTiler.AztecDiamond(size))
        tl = rt.DominoTiler(kernel=int(model == "domino_cftp"), rng=rt.RT_RNG_PHILOX)
    else:
        t = rt.LozengeTiler.MinTiling(rt.LozengeTiler.Hexagon(size, size, size))
        tl = rt.LozengeTiler(kernel=2 if model == "qlozenge" else 0, rng=rt.RT_RNG_PHILOX)
    a = np.array(t, dtype=np.int32)
    tl.Walk(a, 4, 9)
    assert np.array_equal(a, po.walk_fast(model, t, 4, 9))


def test_largest_side_of_two_lattices(monkeypatch):
    import randomtilings_b200 as rt

    monkeypatch.setenv("RT_WALK_KERNEL", "word")
    d = rt.DominoTiler.AztecDiamond(1996)
    tmax, tmin = rt.DominoTiler.MaxTiling(d), rt.DominoTiler.MinTiling(d)
    got, st = rt.DominoTiler(kernel=1, rng=rt.RT_RNG_PHILOX).CFTP(tmax, tmin, first_steps=4, master_seed=5, max_trials=1)
    want, trials, _, ok = po.cftp(tmax, tmin, 4, 5, max_trials=1, fast=True)
    assert (st["trials"], st["coalesced"]) == (trials, ok) == (1, False)
    assert np.array_equal(got, want)
