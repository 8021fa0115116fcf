"""The revaluation split over the dates against the one walk over them (a row budget of one byte), beyond single precision
and beyond the tables that this package's compiler writes.  A book in waves has the bits of the book in one wave, whichever
kernels revalue it."""
from __future__ import annotations

import copy

import numpy as np
import pytest

from oracle import restated
from setups import bermudan, gpu_model, swap_book
from test_gpu_parity import check_sums
from zlatko_b200 import gpu
from zlatko_b200 import spec as S

pytestmark = pytest.mark.gpu

TRADES = [S.Swap(1e6, 0.028, True, S.vanilla_schedule(0.0, 5.0, 2)), S.Forward(0, 5e5, 1.12, 3.0), S.Option(0, True, -4e5, 1.15, 2.0)]
CSA = S.Csa(2e4, 2e4, 5e3)
FIXED_FLOAT, SET_FIXING = 1, 3  # kinds: the low four bits of a record's code


def walked(ctx, run, plan):
    """The plan on revalueKernel, date after date."""
    try:
        ctx.set_row_budget(1)
        return run(plan)
    finally:
        ctx.set_row_budget(0)


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("paths", [64, 129, 4100])
@pytest.mark.parametrize("book", ["swaps", "csa", "bond", "asset", "bermudans"])
def test_double_precision(ctx, book, paths):
    csa = {"csa": CSA, "bermudans": CSA, "bond": S.Csa(2e4, 2e4, 5e3, kind=1, haircut=0.02, bond_maturity=7.0),
           "asset": S.Csa(2e4, 2e4, 5e3, kind=2, haircut=0.05)}.get(book)
    trades = swap_book(6).trades if book == "swaps" else TRADES + ([bermudan(), bermudan(pay=True)] if book == "bermudans" else [])
    p = gpu.compile(gpu_model(paths), S.NettingSet(trades, csa), S.Options(pfe_quantile=0.975))
    if book == "bermudans":
        p = ctx.fit_amc_f64(p)
    got = ctx.run_f64(p)
    assert np.isfinite(got[0]).all() and same(got, walked(ctx, ctx.run_f64, p))


def with_fields(plan, kinds, field):
    """The plan with `field` added to the codes of its records of `kinds`."""
    p = copy.copy(plan)
    p.tables64 = dict(plan.tables64)

    def coded(terms):
        t = terms.reshape(-1, 8).copy()
        hit = np.isin(t[:, 0], kinds)
        assert hit.any()
        t[hit, 0] += field
        return t.reshape(-1)

    p.terms, p.tables64["terms"] = coded(plan.terms), coded(plan.tables64["terms"])
    return p


@pytest.mark.parametrize("kinds", [(FIXED_FLOAT,), (SET_FIXING,), (FIXED_FLOAT, SET_FIXING)])
@pytest.mark.parametrize("field", [1 << 4, 15 << 4, 3 << 12])
@pytest.mark.parametrize("paths", [129, 4100])
def test_fixings_among_the_generic_records(ctx, kinds, field, paths):
    """The trade-group field of a code means nothing outside the per-trade views: a coupon or fixing with a group there is
    priced like the bare one.  It is among the generic records, and a run of dates that starts after the fixing has to find
    it all the same."""
    plan = gpu.compile(gpu_model(paths), S.NettingSet(TRADES, CSA), S.Options(pfe_quantile=0.975))
    p = with_fields(plan, kinds, field)
    got = ctx.run(p)
    assert same(got, walked(ctx, ctx.run, p))
    assert same(ctx.run_f64(p), walked(ctx, ctx.run_f64, p))
    check_sums(p, got[0], restated.run_plan(p)[0], 2e-4)


def rows_and_partials(plans, size=4):
    up = lambda b: (b + 255) // 256 * 256  # noqa: E731
    return sum(up(p.rows_total * p.num_paths * size) + up((p.num_paths + 31) // 32 * p.num_dates * p.stats_per_date * size) for p in plans)


def kernels(ctx, plans):
    b = ctx.batch(plans)
    try:
        return b.info().kernels_per_execute
    finally:
        b.close()


def books(paths, seed=7):
    """Netting sets with Bermudans and margin calls that look back, and one without: the same dates."""
    m = gpu_model(paths, seed)
    m.base_grid = [k / 8.0 for k in range(1, 41)]
    csa = S.Csa(1e4, 1e4, 1e3, 500.0, 0.3)
    return [gpu.compile(m, S.NettingSet(TRADES[:1 + k % 3] + [bermudan(fixed=0.02 + 0.004 * k, pay=bool(k % 2))] * (k > 0), csa),
                        S.Options(collateral_bands=True)) for k in range(4)]


@pytest.mark.parametrize("paths", [1001, 1024])
@pytest.mark.parametrize("slabs", [1, 2, 4])
def test_slabs_within_the_row_budget(ctx, paths, slabs):
    """The values of the split take what the budget leaves beside the rows: slabs of 512 or 256 paths, or the walk."""
    plans = [ctx.fit_amc(p) if p.amc_degrees else p for p in books(paths)]
    tile = len(plans) * plans[0].num_dates * 4 * 256
    rows = rows_and_partials(plans) + len(plans) * 1280  # a byte per path and Bermudan
    whole = ctx.run_many(plans)
    assert kernels(ctx, plans) == 1 + 1 + 3 + 2  # simulate; decide; values with and without Bermudans, settle; statistics
    try:
        ctx.set_row_budget(rows + tile * (4 // slabs) + tile // 2)
        assert kernels(ctx, plans) == 1 + 1 + 3 * slabs + 2
        assert all(same(a, b) for a, b in zip(whole, ctx.run_many(plans)))
        ctx.set_row_budget(rows + tile // 2)
        assert kernels(ctx, plans) == 1 + 1 + 2  # revalueKernel
        assert all(same(a, b) for a, b in zip(whole, ctx.run_many(plans)))
    finally:
        ctx.set_row_budget(0)


@pytest.mark.parametrize("slabs", [1, 2, 4])
def test_slabs_in_double_precision(ctx, slabs):
    p = ctx.fit_amc_f64(books(1001)[1])
    whole = ctx.run_f64(p)
    try:
        ctx.set_row_budget(rows_and_partials([p], 8) + 1280 + p.num_dates * 8 * (256 * (4 // slabs) + 128))
        assert same(whole, ctx.run_f64(p))
    finally:
        ctx.set_row_budget(0)


def test_a_margin_plan_stays_within_the_row_budget(ctx):
    """Plans of the nested margin never run in waves; their split's values count against the budget like the others'."""
    p = gpu.compile(gpu_model(257), S.NettingSet(TRADES, CSA), S.Options(im_quantile=0.99, im_inner_paths=32, im_margin_period=0.25))
    whole = ctx.run(p)
    assert kernels(ctx, [p]) == 1 + 2 + 1 + 2  # simulate; values, settle; the inner paths; statistics
    try:
        ctx.set_row_budget(1)
        assert kernels(ctx, [p]) == 1 + 1 + 1 + 2
        assert same(whole, ctx.run(p))
    finally:
        ctx.set_row_budget(0)


def test_scenarios_share_the_scratch(ctx):
    """Two scenarios in one call, each split over the dates: each has the bits of its own call."""
    plans = [ctx.fit_amc(p) if p.amc_degrees else p for seed in (7, 8) for p in books(777, seed)]
    assert kernels(ctx, plans) == 2 * (1 + 1 + 3) + 2
    both = ctx.run_many(plans)
    for first in (0, 4):
        alone = ctx.run_many(plans[first:first + 4])
        assert all(same(a, b) for a, b in zip(alone, both[first:]))


def test_the_tile_shape_is_the_walks(ctx):
    """A batch that no walk revalues has no tile shape to report; under a row budget it is walked, and tuned."""
    plans = [ctx.fit_amc(p) if p.amc_degrees else p for p in books(20_000)]

    def tile(budget):
        ctx.set_row_budget(budget)
        try:
            b = ctx.batch(plans)
        finally:
            ctx.set_row_budget(0)
        try:
            b.execute()
            return b.info().tile_paths, b.info().num_waves, b.timings()
        finally:
            b.close()

    assert tile(0)[:2] == (256, 1)
    shape, waves, _ = tile(rows_and_partials(plans) // 2)
    assert waves >= 2 and shape in (128, 256, 512)


def test_exercises_out_of_date_order_are_walked(ctx):
    """A plan whose exercise indices do not follow their dates cannot be decided ahead of the values: it takes the walk."""
    p = ctx.fit_amc(books(1001)[1])
    t = p.terms.reshape(-1, 8).copy()
    code = t[:, 0].astype(np.int64)
    hit = np.isin(code & 15, (6, 8, 9))  # policies, and the bonds and coupons after an exercise
    last = (code[hit] >> 12).max()
    t[hit, 0] = (code[hit] & 0xFFF) | ((last - (code[hit] >> 12)) << 12)
    p.terms = t.reshape(-1)
    assert last == 2 and kernels(ctx, [p]) == 1 + 1 + 2
    check_sums(p, ctx.run(p)[0], restated.run_plan(p)[0], 2e-4)
