"""The simulation of many paths (a thread per path or antithetic pair) against that of few (warps with roles): a path's states
follow from its index alone, so the first paths of both have the same bits -- every factor, in both precisions, at the path
counts where the large form begins, odd and even, with and without pairs, foreign rates and credits."""
from __future__ import annotations

import numpy as np
import pytest

from zlatko_b200 import gpu
from zlatko_b200 import spec as S

pytestmark = pytest.mark.gpu

FEW = 999


def plan(paths, antithetic, foreign, credits, substeps):
    asset = S.Asset(1.1, 0.12, S.Curve.flat(0.01))
    if foreign:
        asset.rate_a, asset.rate_sigma = 0.05, 0.01
    n = 2 + foreign + credits
    m = S.Model(curve=S.Curve([1.0, 10.0], [0.02, 0.03]), hw_a=0.05, hw_sigma=0.01, assets=[asset],
                credits=[S.Credit(0.4 + 0.1 * c, 0.02, 0.1, 0.02, [1.0], [0.02], substeps=substeps) for c in range(credits)],
                correlation=np.eye(n) * 0.8 + 0.2, num_paths=paths, seed=7, antithetic=antithetic, base_grid=[0.25, 0.5, 1.0, 2.0])
    return gpu.compile(m, S.NettingSet([S.Forward(0, 5e5, 1.12, 2.0)], None), S.Options(factor_views=True))


@pytest.mark.parametrize("paths,antithetic,foreign,credits,substeps", [
    (37_889, False, 0, 0, 1), (75_777, True, 1, 0, 1), (75_776, True, 0, 0, 1), (75_777, False, 1, 1, 4), (151_553, True, 0, 1, 8),
    (151_553, True, 1, 2, 2), (75_779, False, 0, 2, 1), (265_217, False, 0, 2, 4)])
def test_the_first_paths_are_the_same(ctx, paths, antithetic, foreign, credits, substeps):
    few, many = (plan(n, antithetic, foreign, credits, substeps) for n in (FEW, paths))
    a, b = ctx.run(few, rows=True)[2], ctx.run(many, rows=True)[2]
    assert a.shape[0] >= 3 * few.num_reporting and np.isfinite(b).all()
    assert np.array_equal(a, b[:, :FEW])
    assert not np.array_equal(b[:, -FEW:], b[:, :FEW])  # the last paths are paths of their own
    a, b = ctx.run_f64(few, rows=True)[2], ctx.run_f64(many, rows=True)[2]
    assert np.array_equal(a, b[:, :FEW])
