"""The scratch of the Longstaff-Schwartz fit: bounded, and where a row budget leaves less the realised values are kept in one
row per Bermudan, updated in place, and the Bermudans go in groups or one by one.  The same regressions in another order of
launches: only the order of the sums differs, so the records agree to their single-precision rounding (1e-6 of a record's
scale, 16 units in the last place)."""
from __future__ import annotations

import numpy as np
import pytest

from setups import bermudan, gpu_model
from zlatko_b200 import gpu
from zlatko_b200 import spec as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("basis", ["rate", "rate_swap"])
@pytest.mark.parametrize("rows", [0, 1, 2, 3, 7])  # of realised values; three exercises keep three rows
def test_records_within_the_row_budget(ctx, basis, rows):
    paths = 5000
    trades = [bermudan(fixed=0.015 + 0.004 * k, pay=bool(k % 2), degree=3 - k % 3, basis=basis if k != 2 else "rate",
                       exercise=(1.0, 2.0, 3.0)[k % 2:]) for k in range(6)]
    p = gpu.compile(gpu_model(paths), S.NettingSet(trades, None), S.Options())
    want = ctx.fit_amc(p).terms.reshape(-1, 8).astype(np.float64)
    try:
        ctx.set_row_budget(max(rows * paths * 8, 1))
        got = ctx.fit_amc(p).terms.reshape(-1, 8).astype(np.float64)
    finally:
        ctx.set_row_budget(0)
    scale = np.maximum(np.abs(want), np.abs(want[:, 2:]).max(1, keepdims=True))
    assert np.all(np.abs(got - want) <= 1e-6 * scale + 1e-30)


def test_scratch_is_bounded():
    """16 Bermudans of nine exercises on 500,000 paths: 144 rows of realised values would take 576 MB, the states take 332."""
    import torch

    m = S.Model(curve=S.Curve.flat(0.02), hw_a=0.03, hw_sigma=0.01, num_paths=500_000, seed=3, base_grid=[float(k) for k in range(1, 11)])
    swaps = [S.Swap(1e6, 0.01 + 0.001 * k, bool(k % 2), S.vanilla_schedule(0.0, 10.0, 1)) for k in range(16)]
    p = gpu.compile(m, S.NettingSet([S.Bermudan(s, [float(e) for e in range(1, 10)]) for s in swaps], None), S.Options())
    taken = []
    for budget in (0, 1):
        with gpu.Context(0) as c:
            c.set_row_budget(budget)
            c.amc_states(p, p.exercise_rows)  # the states' own memory
            before = torch.cuda.mem_get_info(0)[0]
            c.fit_amc(p)
            taken.append(before - torch.cuda.mem_get_info(0)[0])
    states = (2 * p.num_dates + p.exercise_rows + p.rows_total) * p.num_paths * 4
    assert taken[0] <= states + (32 << 20)  # the rows, and the partials and the allocator's granularity
    assert taken[1] <= 20 << 20  # one row
