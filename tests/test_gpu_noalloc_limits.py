"""rt_walk_device_noalloc at the last step count that its scratch array holds.  The
bands with halo rows (rt_wordband.cu) have larger exchange slots than the kernel
that exchanges one row (rt_word.cu), which then takes the walk: on one CTA for
lattices of up to 384 words, on the grid for larger ones."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SCRATCH = 16 << 20


def _start(rt, model, size):
    if model == 0:
        return rt.DominoTiler.MinTiling(rt.DominoTiler.AztecDiamond(size))
    return rt.LozengeTiler.MinTiling(rt.LozengeTiler.Hexagon(size, size, size))


# Orders 24 and 60: 364 and 1,984 words; sides 20 and 60.
@pytest.mark.parametrize("model,kernel,size", [(0, 0, 24), (0, 1, 24), (0, 0, 60), (1, 0, 20), (1, 2, 20), (1, 0, 60),
                                               (1, 2, 60)])
def test_last_step_count(model, kernel, size):
    import torch

    import randomtilings_b200 as rt
    from randomtilings_b200 import _capi

    lib = _capi.load()
    cfg = _capi.RtConfig()
    lib.rt_config_default(ctypes.byref(cfg), model)
    cfg.kernel = kernel
    t = np.array(_start(rt, model, size), dtype=np.int32)
    n = int(round(t.size ** 0.5))
    dev = torch.from_numpy(t.copy()).cuda()
    buf = ctypes.create_string_buffer(512)

    def walk(steps):
        return lib.rt_walk_device_noalloc(ctypes.byref(cfg), ctypes.c_void_p(dev.data_ptr()), n, steps, 7, buf, len(buf))

    # The colour arrays take n x n bytes or more; sizes are multiples of 256 bytes,
    # 64 phases, and a walk has steps + 1 phases.
    steps = (SCRATCH - n * n) // 256 * 64 - 1
    while True:
        status = walk(steps)
        if status == _capi.RT_OK:
            break
        assert status == _capi.RT_E_INVAL and b"scratch" in buf.value
        steps -= 64
        assert steps > 0
    want = t.copy()
    (rt.DominoTiler if model == 0 else rt.LozengeTiler)(kernel=kernel).Walk(want, steps, 7)
    assert np.array_equal(dev.cpu().numpy(), want)
