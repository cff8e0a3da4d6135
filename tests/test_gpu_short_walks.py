"""Walks of fewer phases than the planned halo has rows: a band's rows are written
only after the neighbours have read them, so every walk on several CTAs makes an
exchange.  A withheld one ends the walk with a timeout; walks of one step to just
beyond a block of phases, on many CTAs and again and again, equal the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

RT_E_TIMEOUT = -5
REPEATS = 40


def _start(rt, model, size):
    if model == "lozenge":
        return rt.LozengeTiler.MinTiling(rt.LozengeTiler.Hexagon(size, size, size))
    return rt.DominoTiler.MinTiling(rt.DominoTiler.AztecDiamond(size))


def _check(tiler, t, want, steps, seed):
    for _ in range(REPEATS):
        a = np.array(t, dtype=np.int32)
        tiler.Walk(a, steps, seed)
        assert np.array_equal(a, want)


def _withheld(monkeypatch, make, t):
    """The first CTA withholds its rows: its neighbour may not write."""
    import randomtilings_b200 as rt

    monkeypatch.setenv("RT_TEST_DROP_PUBLISH", "0")
    monkeypatch.setenv("RT_WAIT_TIMEOUT_MS", "100")
    a = np.array(t, dtype=np.int32)
    with pytest.raises(rt.RtError) as e:
        make().Walk(a, 1, 3)
    assert e.value.status == RT_E_TIMEOUT


# Order 47: 94 rows; side 40: 81 rows.
@pytest.mark.parametrize("model", ["domino", "lozenge"])
@pytest.mark.parametrize("rng", ["tinymt", "philox"])
def test_word_bands_wait_for_their_neighbours(monkeypatch, model, rng):
    import randomtilings_b200 as rt

    monkeypatch.setenv("RT_WALK_CTAS", "9")
    cls = rt.DominoTiler if model == "domino" else rt.LozengeTiler
    _withheld(monkeypatch, lambda: cls(rng=getattr(rt, f"RT_RNG_{rng.upper()}")),
              _start(rt, model, 47 if model == "domino" else 40))


@pytest.mark.parametrize("model", ["domino", "lozenge"])
@pytest.mark.parametrize("rng", ["tinymt", "philox"])
@pytest.mark.parametrize("ctas", [2, 9, 0])
@pytest.mark.parametrize("steps", [1, 2, 5, 9, 17])
def test_short_word_band_walks(monkeypatch, model, rng, ctas, steps):
    import randomtilings_b200 as rt

    if ctas:
        monkeypatch.setenv("RT_WALK_CTAS", str(ctas))
    t = _start(rt, model, 47 if model == "domino" else 40)
    cls = rt.DominoTiler if model == "domino" else rt.LozengeTiler
    tl = cls(rng=getattr(rt, f"RT_RNG_{rng.upper()}"))
    if rng == "philox":
        want = po.walk_fast(model, t, steps, 11)
    else:
        want = (po.domino_walk if model == "domino" else po.lozenge_walk)(t, steps, 11)
    _check(tl, t, want, steps, 11)


# Order 130: 260 rows; side 90: 270 rows.
@pytest.mark.parametrize("model", ["domino", "lozenge"])
def test_plane_bands_wait_for_their_neighbours(monkeypatch, model):
    import randomtilings_b200 as rt

    monkeypatch.setenv("RT_WALK_CTAS", "12")
    cls = rt.DominoTiler if model == "domino" else rt.LozengeTiler
    _withheld(monkeypatch, lambda: cls(rng=rt.RT_RNG_PLANES), _start(rt, model, 130 if model == "domino" else 90))


@pytest.mark.parametrize("model", ["domino", "lozenge"])
@pytest.mark.parametrize("ctas", [2, 12, 0])
@pytest.mark.parametrize("steps", [1, 3, 20, 33])
def test_short_plane_band_walks(monkeypatch, model, ctas, steps):
    import randomtilings_b200 as rt

    if ctas:
        monkeypatch.setenv("RT_WALK_CTAS", str(ctas))
    t = _start(rt, model, 130 if model == "domino" else 90)
    cls = rt.DominoTiler if model == "domino" else rt.LozengeTiler
    _check(cls(rng=rt.RT_RNG_PLANES), t, po.walk_planes(model, t, steps, 11), steps, 11)


# Bands of more than 2,048 words (rt_plane.cu): order 500 on 5 CTAs, 201 rows of
# 16 words; side 500 on 5, 202 rows of 11 words (12 with padding).
PLANE = {"domino": (500, 5), "lozenge": (500, 5)}


@pytest.mark.parametrize("model", ["domino", "lozenge"])
def test_large_plane_bands_wait_for_their_neighbours(monkeypatch, model):
    import randomtilings_b200 as rt

    size, ctas = PLANE[model]
    monkeypatch.setenv("RT_WALK_CTAS", str(ctas))
    cls = rt.DominoTiler if model == "domino" else rt.LozengeTiler
    _withheld(monkeypatch, lambda: cls(rng=rt.RT_RNG_PLANES), _start(rt, model, size))


@pytest.mark.parametrize("model", ["domino", "lozenge"])
@pytest.mark.parametrize("steps", [1, 6, 8])
def test_short_large_plane_band_walks(monkeypatch, model, steps):
    import randomtilings_b200 as rt

    size, ctas = PLANE[model]
    monkeypatch.setenv("RT_WALK_CTAS", str(ctas))
    t = _start(rt, model, size)
    cls = rt.DominoTiler if model == "domino" else rt.LozengeTiler
    _check(cls(rng=rt.RT_RNG_PLANES), t, po.walk_planes(model, t, steps, 11), steps, 11)


# Bands of four rows with halos of four, and of 7 to 11 rows with halos of four
# and two; one sweep is two pairs of steps.
@pytest.mark.parametrize("n", [90, 333, 1000, 1601])
@pytest.mark.parametrize("sweeps", [1, 2, 3])
def test_short_six_vertex_walks(n, sweeps):
    import randomtilings_b200 as rt

    t = rt.SixVertexTiler()
    h = np.array(rt.SixVertexTiler.MaxHeights(n), dtype=np.int32)
    _check(t, h, np.asarray(po.sixv_walk(h, sweeps, 11)).reshape(-1), sweeps, 11)


@pytest.mark.parametrize("n", [90, 1601])
@pytest.mark.parametrize("sweeps", [1, 40])
def test_six_vertex_bands_wait_for_their_neighbours(monkeypatch, n, sweeps):
    """The first CTA withholds its rows of the first exchange."""
    import randomtilings_b200 as rt

    h = np.array(rt.SixVertexTiler.MaxHeights(n), dtype=np.int32)
    monkeypatch.setenv("RT_TEST_DROP_PUBLISH", "0")
    monkeypatch.setenv("RT_WAIT_TIMEOUT_MS", "100")
    a = h.copy()
    with pytest.raises(rt.RtError) as e:
        rt.SixVertexTiler().Walk(a, sweeps, 3)
    assert e.value.status == RT_E_TIMEOUT
    assert np.array_equal(a, h)


def test_six_vertex_samples_from_epochs_of_one_sweep():
    import randomtilings_b200 as rt

    n, seed = 60, 4
    t = rt.SixVertexTiler()
    got, st = t.CFTP(n, first_sweeps=1, master_seed=seed)
    want, trials, total, ok = po.sixv_cftp(n, 1, seed)
    assert ok and st["coalesced"] and (st["trials"], st["sweeps"]) == (trials, total)
    assert np.array_equal(np.asarray(got).reshape(-1), np.asarray(want).reshape(-1))
