"""A kernel of the MLP that the driver refuses to start (here: it asks for more
shared memory than it may) is an error of the call, and changes no weight."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RT_E_CUDA = -4


def test_refused_launches_are_errors(monkeypatch):
    import randomtilings_b200 as rt
    from randomtilings_b200.mlp import CoordinateMLP

    rng = np.random.default_rng(1)
    x, t = rng.uniform(-1, 1, size=(300, 8)).astype(np.float32), rng.uniform(-1, 1, size=300).astype(np.float32)
    monkeypatch.setenv("RT_TEST_REFUSE_LAUNCH", "1")
    m = CoordinateMLP(seed=4)
    monkeypatch.delenv("RT_TEST_REFUSE_LAUNCH")
    m.set_data(x, t)
    before = m.params
    for call in (lambda: m.predict(x), lambda: m.loss_grad(x, t), lambda: m.train(3, batch=256)):
        with pytest.raises(rt.RtError) as e:
            call()
        assert e.value.status == RT_E_CUDA
    assert np.array_equal(m.params, before)
    # and the device goes on
    n = CoordinateMLP(seed=4)
    n.set_data(x, t)
    assert np.isfinite(n.train(3, batch=256)) and not np.array_equal(n.params, before)
