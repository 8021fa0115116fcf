"""The surrogate's gradient at the edges of its batch split: one 128-row block and less, one block more than the parts of the
weight gradients hold (48 blocks), parts of two blocks with a short last one, the last batch in parts and the first in one chain.  Per parameter block within 5e-3 of the
FP64 oracle at the GPU's bf16 rounding points, the suite's bound for this comparison."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import mlp_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 127, 129, 6144, 6145, 9216, 9217, 40_000])
def test_gradient(ctx, rows):
    from zlatko_b200.surrogate import LAYOUT, Surrogate

    rng = np.random.default_rng(rows)
    x = rng.standard_normal((rows, 16)).astype(np.float32)
    y = (np.sin(x[:, 0]) + 0.5 * x[:, 1] * x[:, 2]).astype(np.float32)
    with Surrogate(ctx, seed=3) as s:
        s.set_params(scaling=np.concatenate([np.zeros(16), np.ones(16), [0.1, 1.3]]).astype(np.float32))
        loss, g = s.gradients(x, y)
        again, g2 = s.gradients(x, y)
        p, sc = s.params()
    assert loss == again and np.array_equal(g, g2)
    want, gw = O.loss_and_grads(p, sc, x, y, emulate=True)
    assert abs(loss - want) <= 1e-3 * want
    o = 0
    for name, shape in LAYOUT:
        k = int(np.prod(shape))
        a, b = g[o:o + k].astype(np.float64), np.asarray(gw[o:o + k], np.float64)
        assert np.linalg.norm(a - b) <= 5e-3 * max(np.linalg.norm(b), 1e-30), name
        o += k
