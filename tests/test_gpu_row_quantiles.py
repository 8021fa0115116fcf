"""The exact row quantile at the edges of its paths: rows shorter than the sampled ones (8K values) and longer, rows that
start off a 16-byte boundary (odd path counts), mostly zero rows (the window overflows), every probability's end.  Against
numpy's order statistics of the GPU's own rows: the quantile interpolates two of the row's values, so it agrees to one
rounding of the interpolation (2 units in the last place)."""
from __future__ import annotations

import numpy as np
import pytest

from setups import gpu_model, gpu_netting_set
from zlatko_b200 import gpu
from zlatko_b200 import spec as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("paths", [1, 2, 255, 4097, 8191, 8192, 8197, 33_333, 100_003])
@pytest.mark.parametrize("level", [0.0, 0.5, 0.975, 1.0])
@pytest.mark.parametrize("csa", [False, True])
def test_exposure_quantiles(ctx, paths, level, csa):
    p = gpu.compile(gpu_model(paths), gpu_netting_set(csa), S.Options(pfe_quantile=level))
    _, values, rows = ctx.run(p, rows=True)
    n = p.num_reporting
    rq = p.requests.reshape(-1, 8)
    checked = 0
    for r in rq:
        if int(r[0]) != 0:
            continue
        row = np.sort(rows[int(r[1])].astype(np.float64))
        h = float(np.float64(r[4])) * (paths - 1)
        k = min(int(np.floor(h)), paths - 1)
        want = row[k] + (h - k) * (row[min(k + 1, paths - 1)] - row[k])
        got = float(values[int(r[7])])
        assert abs(got - want) <= 2 * np.spacing(np.float32(abs(want) + 1e-30)), (int(r[1]), got, want)
        checked += 1
    assert checked >= n
