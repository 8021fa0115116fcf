"""The Longstaff-Schwartz fit at the edges of its launches: fewer paths than a CTA's threads, one path more than a multiple
of them, more Bermudans of one degree and date than share a continuation launch (4), several degrees.  The reference is the
same regression in numpy, in double precision, on the GPU's own states (amc_states): only summation order differs, so the
records agree to their single-precision rounding; tolerance 1e-6 of a record's column scale, 16 units in the last place."""
from __future__ import annotations

import numpy as np
import pytest

from setups import bermudan, gpu_model
from zlatko_b200 import gpu
from zlatko_b200 import spec as S

pytestmark = pytest.mark.gpu


def fit(x, y, degree):
    """center, 1 / scale, c0..c3 by the documented rules."""
    n = x.size
    rec = np.zeros(6)
    rec[1] = 1.0
    if n == 0:
        return rec, lambda v: np.zeros_like(v)
    c, s, d = x.mean(), x.std(), degree
    if s < 1e-12 * max(1.0, abs(c)):
        d = 0
    if n < 2 * (d + 1):
        d = n // 2 - 1 if n >= 4 else 0
    if d == 0:
        rec[:3] = c, 1.0, y.mean()
        return rec, lambda v: np.full_like(v, rec[2])
    A = np.stack([((x - c) / s) ** k for k in range(d + 1)], 1)
    G = A.T @ A + 1e-12 * n * np.eye(d + 1)
    co = np.linalg.solve(G, A.T @ y)
    rec[0], rec[1], rec[2:3 + d] = c, 1.0 / s, co
    return rec, lambda v: np.polyval(co[::-1], (v - c) / s)


@pytest.mark.parametrize("paths", [3, 7, 40, 255, 257, 5000, 37_889])
def test_fit_on_the_gpus_own_states(ctx, paths):
    degrees = [3, 3, 3, 3, 3, 2, 1, 0]
    m = gpu_model(paths)
    trades = [bermudan(fixed=0.015 + 0.004 * k, pay=bool(k % 2), degree=d) for k, d in enumerate(degrees)]
    p = gpu.compile(m, S.NettingSet(trades, None), S.Options())
    got = ctx.fit_amc(p).terms.reshape(-1, 8).astype(np.float64)
    x, D, E = (a.astype(np.float64) for a in ctx.amc_states(p, p.exercise_rows))
    code = p.terms.reshape(-1, 8)[:, 0].astype(np.int64)
    kind, berm, exercise = code & 15, ((code >> 8) & 15) | (((code >> 4) & 15) << 4), code >> 12
    date = np.repeat(np.arange(p.num_dates), np.diff(p.indices[:p.num_dates + 1].astype(np.int64)))
    row, checked = 0, 0
    for b, degree in enumerate(degrees):
        policy = sorted(np.flatnonzero((kind == 6) & (berm == b)), key=lambda t: exercise[t])
        realised = np.zeros(paths)
        want = {}
        for k in range(len(policy) - 1, -1, -1):
            j, e = date[policy[k]], E[row + k]
            itm = e > 0.0
            want[policy[k]], f = fit(x[j][itm], realised[itm] / D[j][itm], degree)
            take = itm & (e > f(x[j]))
            realised = np.where(take, D[j] * e, realised)
            first = date[policy[k - 1]] if k else 0
            for t in np.flatnonzero((kind == 7) & (berm == b)):
                if first <= date[t] < j:
                    want[t], _ = fit(x[date[t]], realised / D[date[t]], degree)
        row += len(policy)
        terms = sorted(want)
        a, w = got[terms][:, 2:], np.array([want[t] for t in terms])
        scale = np.maximum(np.abs(w), np.abs(w[:, 2:]).max(1, keepdims=True) * np.array([0, 0, 1, 1, 1, 1.0]))
        # a cubic through a handful of samples is ill-conditioned: its coefficients carry the rounding of the sums times
        # the condition number, so the smallest samples are held to 1e-4
        assert np.all(np.abs(a - w) <= (1e-6 if paths >= 255 else 1e-4) * scale + 1e-30), b
        checked += len(terms)
    assert checked > 8 * len(degrees) // 2
