"""The MLP's fused gradient kernels at the edges of their row ranges: loss and
gradient against the FP64 restatement, and training that repeats bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import mlp_ref

pytestmark = pytest.mark.gpu


def _batch(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-1, 1, size=(n, 8)).astype(np.float32)
    t = (np.sin(2 * x[:, 0]) * np.cos(3 * x[:, 1]) + 0.3 * x[:, 4]).astype(np.float32)
    return x, t


# One tile; two of a range; ranges of 192 rows (257, 520); a last range without a
# second tile; more ranges than pairs of CTAs (74 x 256 = 18,944).
@pytest.mark.parametrize("n", [2, 127, 128, 129, 256, 257, 384, 520, 1100, 18944, 18945, 40000])
def test_gradient_at_range_edges(n):
    from randomtilings_b200.mlp import CoordinateMLP

    m = CoordinateMLP(seed=4)
    x, t = _batch(n, n)
    loss, g = m.loss_grad(x, t)
    rloss, rg, ry = mlp_ref.loss_grad(m.params, x, t)
    # The restatement rounds to BF16 where the kernels do; what is left is FP32
    # accumulation and BF16 values that round the other way (2^-9 of a value).
    assert abs(loss - rloss) <= 2e-3 * max(1.0, rloss)
    assert np.allclose(m.predict(x), ry, rtol=2e-3, atol=2e-3)
    at = 0
    for name, shape in mlp_ref.SIZES:
        k = int(np.prod(shape))
        a, b = g[at:at + k].astype(np.float64), rg[at:at + k]
        assert np.linalg.norm(a - b) <= 1e-2 * np.linalg.norm(b) + 1e-6, name
        at += k


@pytest.mark.parametrize("batch", [100, 300, 4096])
def test_training_repeats(batch):
    from randomtilings_b200.mlp import CoordinateMLP

    x, t = _batch(5000, 1)
    runs = []
    for _ in range(2):
        m = CoordinateMLP(seed=2)
        m.set_data(x, t)
        loss = m.train(20, batch=batch, seed=3)
        runs.append((loss, m.params))
    assert runs[0][0] == runs[1][0]
    assert np.array_equal(runs[0][1], runs[1][1])
