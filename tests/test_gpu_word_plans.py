"""The word kernel's launch shapes (rt_word.cu) against the oracle: one CTA,
one thread-block cluster (rows exchanged through distributed shared memory)
and the cooperative grid, at the edges of the planner's ranges; runs of
same-colour steps cut by epochs and by a full schedule buffer."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _walk(tiler, t, steps, seed):
    a = np.array(t, dtype=np.int32)
    tiler.Walk(a, steps, seed)
    return a


def _aztec(order):
    import randomtilings_b200 as rt

    return rt.DominoTiler.MaxTiling(rt.DominoTiler.AztecDiamond(order))


def _hexagon(*sides):
    import randomtilings_b200 as rt

    return rt.LozengeTiler.MaxTiling(rt.LozengeTiler.Hexagon(*sides))


# Rows x words of a row: order 25 54 x 7 = 378 (the last on one CTA), 26 56 x 8
# = 448; 135 274 x 35 = 9,590 (the last on one cluster), 136 9,660.
@pytest.mark.parametrize("order", [2, 25, 26, 135, 136, 256])
@pytest.mark.parametrize("cftp", [False, True])
def test_domino_planner_edges(order, cftp):
    import randomtilings_b200 as rt

    t = _aztec(order)
    got = _walk(rt.DominoTiler(kernel=int(cftp)), t, 500, 11)
    assert np.array_equal(got, po.domino_walk(t, 500, 11, cftp=cftp))


# 330, 378 (one CTA); 432, 9,408 (one cluster); 9,831 words.
@pytest.mark.parametrize("sides", [(2, 1, 3), (27, 30, 26), (28, 33, 30), (166, 163, 160), (170, 160, 150)])
@pytest.mark.parametrize("rng", [0, 1])
def test_lozenge_planner_edges(sides, rng):
    import randomtilings_b200 as rt

    t = _hexagon(*sides)
    got = _walk(rt.LozengeTiler(rng=rng), t, 500, 12)
    want = po.walk_fast("lozenge", t, 500, 12) if rng else po.lozenge_walk(t, 500, 12)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("ctas", [2, 5, 15, 16, 17, 40])
def test_cluster_and_grid_sizes(monkeypatch, ctas):
    """Bands of one to nineteen rows, a last band shorter than the others."""
    import randomtilings_b200 as rt

    monkeypatch.setenv("RT_WALK_CTAS", str(ctas))
    t = _aztec(17)
    assert np.array_equal(_walk(rt.DominoTiler(), t, 700, 3), po.domino_walk(t, 700, 3))
    t = _hexagon(13, 18, 9)
    assert np.array_equal(_walk(rt.LozengeTiler(kernel=2), t, 700, 4), po.lozenge_walk(t, 700, 4, qweight=True))


@pytest.mark.parametrize("ctas", [1, 4, 20])
def test_coupled_chains_and_epochs(monkeypatch, ctas):
    """CFTP walks both chains through every epoch: an epoch that begins with
    the colour the last one ended with has no Update pending."""
    import randomtilings_b200 as rt

    monkeypatch.setenv("RT_WALK_CTAS", str(ctas))
    d = rt.DominoTiler.AztecDiamond(12)
    tmax, tmin = rt.DominoTiler.MaxTiling(d), rt.DominoTiler.MinTiling(d)
    got, st = rt.DominoTiler(kernel=1).CFTP(tmax, tmin, first_steps=16, master_seed=5, max_trials=20)
    want, _, total, ok = po.cftp(tmax, tmin, 16, 5, max_trials=20)
    assert ok and st["coalesced"] and st["total_steps"] == total
    assert np.array_equal(got, want)


@pytest.mark.parametrize("steps", [1, 4095, 4096, 7001])
def test_noalloc_schedule_buffer(steps):
    """rt_walk_device_noalloc stages its runs 2,048 at a time."""
    import ctypes

    import torch

    import randomtilings_b200 as rt
    from randomtilings_b200 import _capi

    lib = _capi.load()
    for model, t, want in ((rt.RT_DOMINO, _aztec(9), po.domino_walk), (rt.RT_LOZENGE, _hexagon(5, 6, 4), po.lozenge_walk)):
        cfg = _capi.RtConfig()
        lib.rt_config_default(ctypes.byref(cfg), model)
        n = int(round(len(t) ** 0.5))
        d = torch.tensor(np.array(t, dtype=np.int32), device="cuda")
        torch.cuda.synchronize()
        _capi.check(lib.rt_walk_device_noalloc(ctypes.byref(cfg), d.data_ptr(), n, steps, 6, None, 0))
        assert np.array_equal(d.cpu().numpy(), want(t, steps, 6))
