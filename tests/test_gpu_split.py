"""The revaluation split over the dates against the one walk over them: a row budget of one byte runs every netting set
in a wave of its own on revalueKernel, without it the same plans run on decideKernel, valueKernel and settleKernel.  Both
take the same arithmetic and the same statistics tree, so the results are the same bits: edges of the path tiles (32, 64,
128, 256), of the dates held at a time, every collateral form, Bermudans in registers and in bytes, exercise rows."""
from __future__ import annotations

import numpy as np
import pytest

from setups import bermudan, gpu_model
from zlatko_b200 import gpu
from zlatko_b200 import spec as S

pytestmark = pytest.mark.gpu

SWAP = S.Swap(1e6, 0.028, True, S.vanilla_schedule(0.0, 5.0, 2))
TRADES = [SWAP, S.Forward(0, 5e5, 1.12, 3.0), S.Option(0, True, -4e5, 1.15, 2.0)]


def both(ctx, plans):
    ctx.set_basis(ctx.BASIS_OFF)
    try:
        split = ctx.run_many(plans)
        ctx.set_row_budget(1)
        walk = ctx.run_many(plans)
    finally:
        ctx.set_row_budget(0)
        ctx.set_basis(ctx.BASIS_AUTO)
    for (s0, v0), (s1, v1) in zip(split, walk):
        assert np.isfinite(s0).all()
        assert np.array_equal(s0, s1) and np.array_equal(v0, v1)


@pytest.mark.parametrize("paths", [1, 31, 33, 64, 127, 129, 255, 1001, 2048])
@pytest.mark.parametrize("csa", [None, S.Csa(2e4, 2e4, 5e3), S.Csa(2e4, float("inf"), 5e3), S.Csa(1e4, 1e4, 1e3, 500.0, 0.3),
                                 S.Csa(2e4, 2e4, 5e3, kind=1, haircut=0.02, bond_maturity=7.0),
                                 S.Csa(2e4, 2e4, 5e3, kind=2, haircut=0.05)])
def test_one_netting_set(ctx, paths, csa):
    m = gpu_model(paths)
    both(ctx, [gpu.compile(m, S.NettingSet(TRADES, csa), S.Options(pfe_quantile=0.975, collateral_bands=csa is not None, gross=False,
                                                                  im_quantile=0.99))])


@pytest.mark.parametrize("dates", [1, 31, 32, 33, 64, 65])
def test_dates_held_at_a_time(ctx, dates):
    m = gpu_model(777)
    m.base_grid = [k / 16.0 for k in range(1, dates + 1)]
    both(ctx, [gpu.compile(m, S.NettingSet([S.Swap(1e6, 0.028, True, [0.0, dates / 16.0])], None), S.Options())])


@pytest.mark.parametrize("paths,sets", [(4097, 12), (2368, 12), (2369, 12), (9000, 40)])
def test_many_netting_sets(ctx, paths, sets):
    m = gpu_model(paths)
    both(ctx, [gpu.compile(m, S.NettingSet(TRADES * (1 + k % 3), S.Csa(1e4 * k, 1e4 * k, 5e3)), S.Options()) for k in range(sets)])


@pytest.mark.parametrize("count,basis", [(1, "rate"), (3, "rate"), (6, "rate"), (2, "rate_swap")])
@pytest.mark.parametrize("paths", [500, 4099])
def test_bermudans(ctx, count, basis, paths):
    m = gpu_model(paths)
    ex = [bermudan(fixed=0.02 + 0.004 * k, pay=bool(k % 2), physical=k != 1, basis=basis) for k in range(count)]
    p = gpu.compile(m, S.NettingSet(TRADES + ex, S.Csa(2e4, 2e4, 5e3)), S.Options(exercise_views=count <= 4))
    p = ctx.fit_amc(p)
    q = gpu.compile(m, S.NettingSet(TRADES, S.Csa(2e4, 2e4, 5e3)), S.Options())  # a lean plan of the same launch
    both(ctx, [p, q] if q.num_dates == p.num_dates else [p])
