"""The simulate kernel at the edges of its shapes: CTAs of 32 or 64 paths (antithetic pairs, up to 18,944 paths and
beyond) or of 32 unpaired paths, zero to two CIR++ credits (producer warps), one sub-step or several (dates per ring
buffer), against the restated FP32 kernels.  Tolerance: 2e-4 of a statistic's scale, the suite's bound for FP32 plans."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import restated
from setups import gpu_netting_set
from zlatko_b200 import gpu
from zlatko_b200 import spec as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    with gpu.Context(0) as c:
        yield c


@pytest.mark.parametrize("paths,antithetic,credits,substeps", [
    (1, True, 1, 4), (2, True, 2, 4), (31, True, 0, 1), (33, True, 1, 1), (64, True, 2, 1), (65, False, 1, 4), (127, False, 0, 1),
    (1000, False, 2, 8), (1001, True, 2, 8), (18_944, True, 1, 4), (18_945, True, 1, 4), (19_007, True, 0, 1),
    (19_010, True, 2, 1), (18_945, False, 1, 4)])
def test_simulation_matches_the_restated_kernels(ctx, paths, antithetic, credits, substeps):
    cr = [S.Credit(0.4 + 0.1 * c, 0.02, 0.1, 0.02, [1.0], [0.02], substeps=substeps) for c in range(credits)]
    f = 2 + credits
    corr = np.eye(f) + 0.2 * (np.eye(f, k=1) + np.eye(f, k=-1))
    m = S.Model(curve=S.Curve([1.0, 10.0], [0.02, 0.03]), hw_a=0.05, hw_sigma=0.01, assets=[S.Asset(1.1, 0.12, S.Curve.flat(0.01))],
                credits=cr, correlation=corr, num_paths=paths, seed=7, antithetic=antithetic, base_grid=[k / 4.0 for k in range(1, 21)])
    plan = gpu.compile(m, gpu_netting_set(False), S.Options())
    got, _ = ctx.run(plan)
    want, _ = restated.run_plan(plan)
    n = plan.stats_per_date
    g, w = got.reshape(-1, n).astype(np.float64), want.reshape(-1, n).astype(np.float64)
    assert np.isfinite(g).all()
    for k in range(n):
        scale = max(np.abs(w[:, k]).max(), 1e-6 * np.abs(w).max())
        assert np.abs(g[:, k] - w[:, k]).max() <= 2e-4 * scale, k
