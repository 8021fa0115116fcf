"""The revaluation split over the dates against the one walk over them (a row budget of one byte), beyond single precision
and beyond the tables that this package's compiler writes.  A book in waves has the bits of the book in one wave, whichever
kernels revalue it."""
from __future__ import annotations

import numpy as np
import pytest

from setups import bermudan, gpu_model, swap_book
from zlatko_b200 import gpu
from zlatko_b200 import spec as S

pytestmark = pytest.mark.gpu

TRADES = [S.Swap(1e6, 0.028, True, S.vanilla_schedule(0.0, 5.0, 2)), S.Forward(0, 5e5, 1.12, 3.0), S.Option(0, True, -4e5, 1.15, 2.0)]
CSA = S.Csa(2e4, 2e4, 5e3)


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
