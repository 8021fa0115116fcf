"""The reduction of the partials: a single-precision overflow of the last 128 paths leaves its statistic infinite."""
from __future__ import annotations

import numpy as np
import pytest

from setups import gpu_model
from zlatko_b200 import gpu
from zlatko_b200 import spec as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("paths", [100, 128])
def test_an_infinite_statistic_of_one_group(ctx, paths):
    p = gpu.compile(gpu_model(paths), S.NettingSet([S.Forward(0, 3e38, 0.5, 3.0)], None), S.Options())
    sums = ctx.run(p)[0].reshape(-1, p.stats_per_date)
    held = p.times < 3.0
    assert np.isposinf(sums[held, 0]).all() and np.isposinf(sums[held, 1]).all()  # E[V], E[max(V, 0)]
    assert np.isfinite(sums[:, 6:8]).all()  # survival, discount factor
