"""The exact row quantile where the sample's window fills the pool of kept values (median of 250,000 to 350,000 values), holds
more than it (longer rows, equal values: no window pass) and little of it, in both precisions.  Against numpy's order
statistics of the GPU's own rows: the interpolation's rounding, 2 units in the last place of the row's type."""
from __future__ import annotations

import numpy as np
import pytest

from setups import gpu_model
from zlatko_b200 import gpu
from zlatko_b200 import spec as S

pytestmark = pytest.mark.gpu

BOOKS = {"swap": ([S.Swap(1e6, 0.028, True, S.vanilla_schedule(0.0, 5.0, 2)), S.Forward(0, 5e5, 1.12, 3.0)], None),
         "mostly zero": ([S.Option(0, True, 4e5, 1.6, 2.0)], None),
         "collateralised": ([S.Forward(0, 5e5, 1.12, 3.0)], S.Csa(0.0, 0.0, 0.0))}


@pytest.mark.parametrize("book", list(BOOKS))
@pytest.mark.parametrize("paths", [262_144, 330_001, 1_000_003])
@pytest.mark.parametrize("level", [0.5, 0.9, 0.975, 0.999])
@pytest.mark.parametrize("f64", [False, True])
def test_quantiles_of_long_rows(ctx, book, paths, level, f64):
    m = gpu_model(paths)
    m.base_grid = [0.5, 2.0]
    p = gpu.compile(m, S.NettingSet(*BOOKS[book]), S.Options(pfe_quantile=level))
    _, values, rows = ctx.run_f64(p, rows=True) if f64 else ctx.run(p, rows=True)
    eps = np.spacing if f64 else lambda v: np.spacing(np.float32(v))
    checked = 0
    for r in (p.tables64["requests"] if f64 else p.requests).reshape(-1, 8):
        if int(r[0]) != 0:
            continue
        h = float(r[4]) * (paths - 1)
        k = min(int(np.floor(h)), paths - 1)
        k1 = min(k + 1, paths - 1)
        row = np.partition(rows[int(r[1])].astype(np.float64), (k, k1))
        want = row[k] + (h - k) * (row[k1] - row[k])
        assert abs(float(values[int(r[7])]) - want) <= 2 * eps(abs(want) + 1e-30), int(r[1])
        checked += 1
    assert checked == p.num_reporting
