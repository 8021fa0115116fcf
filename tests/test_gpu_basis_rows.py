"""The basis kernel's exposure rows and statistics at path counts around its stores and its tile (128 paths, units of 32, rows
written 8 paths, 4 paths or one path at a time), against the term-by-term kernel on the same normals.

Tolerances as for the same comparison at one size (tests/test_gpu_basis.py): a value agrees to 1e-4 of the rows' scale unless
its path's margin call sits on the boundary of the transfer rule (at most 1% of the paths, or one), the median to 1e-6."""
import numpy as np
import pytest

from zlatko_b200 import gpu, workloads
from zlatko_b200 import spec as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("paths", [1, 8, 33, 127, 128, 136, 1001, 1004, 4096])
def test_rows_at_every_store_width(ctx, paths):
    m, books, o, _ = workloads.correlated_csa_book(paths, netting_sets=30, num_trades=450, foreign_rates=True)
    csas = [None, S.Csa(1e5, 1e5, 1e4, 0.0, 10.0 / 250.0), S.Csa(2e5, -1.0, 0.0, 5e4, 10.0 / 250.0)]
    plans = [gpu.compile(m, S.NettingSet(b.trades, csa) if csa else S.NettingSet(b.trades), o) for b, csa in zip(books, csas)]
    for i, p in enumerate(plans):
        got = []
        for mode in (gpu.Context.BASIS_ALL, gpu.Context.BASIS_OFF):
            ctx.set_basis(mode)
            try:
                got.append(ctx.run(p, rows=True))
            finally:
                ctx.set_basis(gpu.Context.BASIS_AUTO)
        H = p.header
        a, b = (r[2][H[28]:H[28] + len(p.reporting)].astype(np.float64) for r in got)
        scale = max(np.abs(b).max(), 1.0)
        moved = (np.abs(a - b) > 1e-4 * scale).any(axis=0)
        assert moved.sum() <= (max(1, paths // 100) if csas[i] else 0), (i, moved.sum())
        assert np.median(np.abs(a - b)) <= 1e-6 * scale, i
