"""A handle's launch plan is the plan of the walk it launches: a walk that cannot
be planned leaves the handle as it was, and nothing of one lattice's plan is left
in the next one's."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu


def _walk(tiler, t, steps, seed):
    a = np.array(t, dtype=np.int32)
    tiler.Walk(a, steps, seed)
    return a


def _aztec(rt, order):
    return rt.DominoTiler.MinTiling(rt.DominoTiler.AztecDiamond(order))


@pytest.mark.parametrize("kernel", ["", "word", "generic"])
def test_walks_go_on_after_one_that_cannot_be_planned(monkeypatch, kernel):
    """Side 8,000 has too many generator states for any kernel."""
    import randomtilings_b200 as rt

    if kernel:
        monkeypatch.setenv("RT_WALK_KERNEL", kernel)
    t = _aztec(rt, 47)
    tl = rt.DominoTiler()
    want = po.domino_walk(t, 60, 5)
    assert np.array_equal(_walk(tl, t, 60, 5), want)
    with pytest.raises(rt.RtError):
        tl.Walk(np.zeros(8000 * 8000, dtype=np.int32), 4, 5)
    assert np.array_equal(_walk(tl, t, 60, 5), want)


@pytest.mark.parametrize("ctas", [7, 12])
@pytest.mark.parametrize("orders", [(130, 24), (24, 130), (130, 24, 130)])
def test_one_handle_walks_large_and_small_lattices(monkeypatch, ctas, orders):
    import randomtilings_b200 as rt

    monkeypatch.setenv("RT_WALK_CTAS", str(ctas))
    tl = rt.DominoTiler()
    for order in orders:
        t = _aztec(rt, order)
        assert np.array_equal(_walk(tl, t, 60, 5), po.domino_walk(t, 60, 5))


def _cases(rt):
    D, L, R, T = rt.DominoTiler, rt.LozengeTiler, rt.RectTriangleTiler, rt.TriangleDimerTiler
    philox, planes = rt.RT_RNG_PHILOX, rt.RT_RNG_PLANES
    return {
        "word bands": (lambda: D(rng=philox), [_aztec(rt, 200), _aztec(rt, 8)]),
        "words": (lambda: D(rng=philox), [_aztec(rt, 900), _aztec(rt, 520)]),
        "plane bands": (lambda: D(rng=planes), [_aztec(rt, 900), _aztec(rt, 8)]),
        "rectangle-triangles": (lambda: R(rng=philox), [R.maxHex(60), R.maxHex(40)]),
        "triangle dimers": (lambda: T(rng=philox), [T.BiboneHexagon(64), T.BiboneHexagon(9)]),
        "triangle dimers, bit-exact": (lambda: T(), [T.BiboneHexagon(64), T.BiboneHexagon(9)]),
    }


@pytest.mark.parametrize("kind", ["word bands", "words", "plane bands", "rectangle-triangles", "triangle dimers",
                                  "triangle dimers, bit-exact"])
def test_handles_of_unequal_sizes_in_turn(kind):
    """A handle's plan stays good while another handle plans a smaller lattice for
    the same kernel."""
    import randomtilings_b200 as rt

    make, (large, small) = _cases(rt)[kind]
    large, small = np.asarray(large, dtype=np.int32), np.asarray(small, dtype=np.int32)
    alone = make()
    want = _walk(alone, large, 40, 5)
    alone.close()
    a, b = make(), make()
    assert np.array_equal(_walk(a, large, 40, 5), want)
    _walk(b, small, 40, 5)
    assert np.array_equal(_walk(a, large, 40, 5), want)
