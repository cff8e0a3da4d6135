"""The fast mode's word kernel on bands with halos (rt_wordband.cu) against the
oracle: one CTA to many, halos of four to sixteen rows (blocks that are and are
not a multiple of the colour round), uneven bands, bands of too few rows (which
rt_word.cu takes), the widest bands with four halo rows, and two lattices."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _walk(tiler, t, steps, seed):
    a = np.array(t, dtype=np.int32)
    tiler.Walk(a, steps, seed)
    return a


def _start(rt, model, *size):
    if model in ("domino", "domino_cftp"):
        return rt.DominoTiler.MinTiling(rt.DominoTiler.AztecDiamond(*size))
    return rt.LozengeTiler.MinTiling(rt.LozengeTiler.Hexagon(*size))


def _tiler(rt, model):
    if model in ("domino", "domino_cftp"):
        return rt.DominoTiler(kernel=int(model == "domino_cftp"), rng=rt.RT_RNG_PHILOX, chain=4)
    return rt.LozengeTiler(kernel=2 if model == "qlozenge" else 0, rng=rt.RT_RNG_PHILOX, chain=4)


@pytest.mark.parametrize("model", ["domino", "domino_cftp", "lozenge", "qlozenge"])
@pytest.mark.parametrize("ctas", [0, 1, 2, 5, 9, 13, 24, 60])
def test_walks_match_the_oracle(monkeypatch, model, ctas):
    import randomtilings_b200 as rt

    if ctas:
        monkeypatch.setenv("RT_WALK_CTAS", str(ctas))
    t = _start(rt, model, *((47,) if model.startswith("domino") else (40, 55, 31)))
    assert np.array_equal(_walk(_tiler(rt, model), t, 151, 2**33 + 5), po.walk_fast(model, t, 151, 2**33 + 5, chain=4))


@pytest.mark.parametrize("model,size", [("domino", (7,)), ("domino", (300,)), ("domino_cftp", (340,)),
                                        ("lozenge", (5, 6, 4)), ("qlozenge", (300, 290, 310))])
def test_edges_of_the_plan(model, size):
    import randomtilings_b200 as rt

    t = _start(rt, model, *size)
    assert np.array_equal(_walk(_tiler(rt, model), t, 40, 77), po.walk_fast(model, t, 40, 77, chain=4))


@pytest.mark.parametrize("ctas", [1, 3, 6])
def test_two_lattices(monkeypatch, ctas):
    import randomtilings_b200 as rt

    monkeypatch.setenv("RT_WALK_CTAS", str(ctas))
    d = rt.DominoTiler.AztecDiamond(12)
    tmax, tmin = rt.DominoTiler.MaxTiling(d), rt.DominoTiler.MinTiling(d)
    got, st = rt.DominoTiler(kernel=1, rng=rt.RT_RNG_PHILOX).CFTP(tmax, tmin, first_steps=16, master_seed=5, max_trials=20)
    want, trials, total, ok = po.cftp(tmax, tmin, 16, 5, max_trials=20, fast=True)
    assert ok and st["coalesced"] and (st["trials"], st["total_steps"]) == (trials, total)
    assert np.array_equal(got, want)
