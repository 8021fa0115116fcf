"""The work that users of this package give it: what it is, over which sizes, and what it has to return.

Every case is one of five kinds of work, at the sizes of the package's own workloads, tests and benchmark:

    book     netting sets of swaps, FX forwards and FX options revalued on simulated paths: the exposure statistics
             (EE, ENE, EE*, CVA increments, ...) and the PFE of every netting set and date, through Context.run /
             run_many (host tables in, host statistics out), Context.run_f64, or a resident Batch
    amc      Bermudan swaptions: the Longstaff-Schwartz fit alone (Context.fit_amc), or the fit and the exposure run
    mixed    a book with 5% Bermudans, each netting set with and without its CSA, as a resident Batch
    margin   the conditional initial margin of a netting set by nested Monte Carlo
    net      the revaluation surrogate: the gradient of one batch, or the predictions of many rows

listed() names the cases, draw() gives more of the same ranges.  Portfolios, models and simulation seeds follow from
the case and the seed alone.  exact() restates the plans' semantics in plain torch, in 64 bits: it reads the tables
that a program hands over (the plan) and shares no code with the kernels.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from zlatko_b200 import gpu, workloads
from zlatko_b200 import spec as S
from zlatko_b200.surrogate import Surrogate

PFE = 0.975
MPR = 10.0 / 250.0  # ten business days between a margin call's valuation and its date


# ---------------------------------------------------------------------------------------------------------------
# The cases

def _book(name, call, paths, sets, trades, months, csa, foreign, swaps_only=False):
    return {"name": name, "kind": "book", "call": call, "paths": paths, "sets": sets, "trades": trades, "months": months,
            "csa": csa, "foreign": foreign, "swaps_only": swaps_only}


def listed():
    return [
        # A trader asks for one small collateralised netting set before a trade: latency is all that counts.
        _book("what_if", "run", 2_000, 1, 3, 60, True, False),
        # The uncollateralised swap portfolio of the package's first workload: 20 swaps, 10,000 paths, 60 months.
        _book("swaps", "run", 10_000, 1, 20, 60, False, False, swaps_only=True),
        # The same portfolio in the FP64 mode, which validation runs use.
        _book("swaps_f64", "f64", 10_000, 1, 20, 60, False, False, swaps_only=True),
        # A desk of a dozen counterparties, an odd path count and a horizon of seven years.
        _book("desk", "run", 33_333, 12, 119, 84, True, True),
        # The correlated CSA book of the package's second workload, as one call from host tables.
        _book("csa_book", "run", 100_000, 100, 1_000, 120, True, True),
        # The benchmark's book (2,000 trades in 100 netting sets) resident on the device, on half a million paths.
        _book("large_book", "batch", 500_000, 100, 2_000, 120, True, True),
        # The Longstaff-Schwartz fit of one netting set of the Bermudan workload (200,000 paths, 40 dates).
        {"name": "amc_fit", "kind": "amc", "call": "fit", "paths": 200_000, "bermudans": 4, "sets": 1, "basis": "rate"},
        # Bermudans on the two-regressor basis, from the compiled plans to the exposure.
        {"name": "amc_two", "kind": "amc", "call": "fit_run", "paths": 50_000, "bermudans": 6, "sets": 2, "basis": "rate_swap"},
        # A slice of the large XVA batch: Bermudans among swaps, forwards and options, with and without CSA.
        {"name": "mixed", "kind": "mixed", "paths": 65_536, "sets": 24, "trades": 800},
        # The conditional initial margin (128 inner paths) of a netting set of 100 trades.
        {"name": "margin", "kind": "margin", "paths": 10_000, "trades": 100, "months": 60, "inner": 128},
        # One training batch of the surrogate: loss and gradient.
        {"name": "net_gradients", "kind": "net", "call": "gradients", "rows": 8_192},
        # Revaluation by the surrogate from host rows.
        {"name": "net_predict", "kind": "net", "call": "predict", "rows": 262_144},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["book", "book", "book", "book", "amc", "amc", "mixed", "margin", "net", "net"])
    if kind == "book":
        call = rng.choice(["run", "run", "batch", "f64"])
        swaps_only = rng.random() < 0.25
        if call == "f64":
            c = _book("", call, _log(rng, 500, 30_000), 1, rng.randint(1, 60), rng.randint(12, 120), rng.random() < 0.5,
                      rng.random() < 0.5, swaps_only)
        else:
            sets = _log(rng, 1, 100)
            c = _book("", call, _log(rng, 1_000, 200_000), sets, sets + _log(rng, 1, 900), rng.randint(24, 120),
                      rng.random() < 0.7, rng.random() < 0.6, swaps_only)
        del c["name"]
        return c
    if kind == "amc":
        basis = rng.choice(["rate", "rate", "rate_swap"])
        sets = rng.randint(1, 3)
        return {"kind": kind, "call": "fit" if basis == "rate" and rng.random() < 0.5 else "fit_run",
                "paths": _log(rng, 2_000, 200_000), "bermudans": sets * rng.randint(1, 4), "sets": sets, "basis": basis}
    if kind == "mixed":
        sets = rng.randint(4, 30)
        return {"kind": kind, "paths": _log(rng, 4_000, 65_536), "sets": sets, "trades": sets * rng.randint(4, 33)}
    if kind == "margin":
        return {"kind": kind, "paths": _log(rng, 500, 10_000), "trades": rng.randint(2, 150), "months": rng.randint(12, 72),
                "inner": rng.randint(32, 160)}
    call = rng.choice(["gradients", "predict"])
    return {"kind": kind, "call": call, "rows": _log(rng, 200, 131_072) if call == "gradients" else _log(rng, 500, 1_000_000)}


# ---------------------------------------------------------------------------------------------------------------
# Portfolios and models, from the case and the seed

def _trades(rng, n, months, spots, swaps_only):
    """The workloads' 60/30/10 mix of swaps, FX forwards and FX options, nothing longer than the horizon."""
    out = []
    n_swaps = n if swaps_only else max(1, round(0.6 * n))
    n_fwds = 0 if swaps_only else min(n - n_swaps, round(0.3 * n))
    for k in range(n):
        if k < n_swaps:
            out.append(workloads.random_swap(rng, months))
            continue
        a = int(rng.integers(0, 2))
        strike = spots[a] * rng.uniform(0.9, 1.1)
        sign = rng.choice([-1.0, 1.0])
        if k < n_swaps + n_fwds:
            out.append(S.Forward(a, sign * rng.uniform(1e6, 1e7), strike, int(rng.integers(3, min(61, months + 1))) / 12.0))
        else:
            out.append(S.Option(a, bool(rng.random() < 0.5), sign * rng.uniform(1e6, 5e6), strike,
                                int(rng.integers(3, min(37, months + 1))) / 12.0))
    return [out[i] for i in rng.permutation(n)]


def _model(rng, case, months, foreign):
    """Domestic Hull-White rate, two lognormal FX rates, a CIR++ intensity, and with `foreign` two foreign Hull-White
    rates, joined by a correlation with off-diagonals U[-0.3, 0.5] projected to the nearest correlation matrix."""
    spots = (1.1, 0.9)
    fx = [S.Asset(s, rng.uniform(0.08, 0.15), S.Curve.flat(rng.uniform(0.0, 0.04))) for s in spots]
    if foreign:
        for a in fx:
            a.rate_a, a.rate_sigma = rng.uniform(0.01, 0.1), rng.uniform(0.005, 0.015)
    f = 6 if foreign else 4
    c = np.eye(f)
    iu = np.triu_indices(f, 1)
    c[iu] = rng.uniform(-0.3, 0.5, size=len(iu[0]))
    c = workloads.nearest_correlation(np.triu(c) + np.triu(c, 1).T)
    return S.Model(curve=S.Curve.flat(0.02), hw_a=rng.uniform(0.01, 0.1), hw_sigma=rng.uniform(0.005, 0.015), assets=fx,
                   credits=[S.Credit(0.5, 0.02, 0.08, 0.02, [1.0], [0.01], substeps=8)], correlation=c,
                   num_paths=case["paths"], seed=int(rng.integers(1, 1 << 31)), antithetic=True,
                   base_grid=[k / 12.0 for k in range(1, months + 1)])


def _csa(rng):
    t = rng.uniform(0.0, 5e6)
    return S.Csa(t, t, 1e5, 0.0, MPR)


def _sets(rng, case, trades, csa):
    books, at = [], 0
    for n in workloads.zipf_sizes(len(trades), case["sets"], 1.2):
        books.append(S.NettingSet(trades[at:at + n], _csa(rng) if csa else None))
        at += n
    return books


def _bermudan(rng, basis):
    atm = float(np.expm1(0.02))
    return S.Bermudan(S.Swap(1e7, atm + rng.uniform(-0.01, 0.01), bool(rng.random() < 0.5), S.vanilla_schedule(0.0, 10.0, 1)),
                      [float(e) for e in range(1, 10)], physical=True, position=1.0, degree=3, basis=basis)


def _plans(case, seed):
    """The case's compiled plans; Bermudans are not fitted yet."""
    rng = np.random.default_rng([seed, 20261205])
    if case["kind"] == "book":
        if case["swaps_only"] and not case["foreign"]:  # the swap portfolio: one short rate, a flat hazard
            m = S.Model(curve=S.Curve.flat(0.02), hw_a=0.03, hw_sigma=0.01,
                        credits=[S.Credit(1e-6, 0.0, 0.0, 0.0, [1.0], [0.01], substeps=1)], num_paths=case["paths"],
                        seed=int(rng.integers(1, 1 << 31)), antithetic=True,
                        base_grid=[k / 12.0 for k in range(1, case["months"] + 1)])
            spots = (1.0, 1.0)
        else:
            m = _model(rng, case, case["months"], case["foreign"])
            spots = [a.spot for a in m.assets]
        trades = _trades(rng, case["trades"], case["months"], spots, case["swaps_only"])
        return [gpu.compile(m, b, S.Options(pfe_quantile=PFE)) for b in _sets(rng, case, trades, case["csa"])]
    if case["kind"] == "amc":
        m = S.Model(curve=S.Curve.flat(0.02), hw_a=0.03, hw_sigma=0.01, num_paths=case["paths"],
                    seed=int(rng.integers(1, 1 << 31)), antithetic=True, base_grid=[k / 4.0 for k in range(1, 41)])
        per = case["bermudans"] // case["sets"]
        return [gpu.compile(m, S.NettingSet([_bermudan(rng, case["basis"]) for _ in range(per)], None), S.Options(pfe_quantile=PFE))
                for _ in range(case["sets"])]
    if case["kind"] == "mixed":
        m = _model(rng, case, 120, True)
        spots = [a.spot for a in m.assets]
        n_berm = max(1, case["trades"] // 20)
        trades = _trades(rng, case["trades"] - n_berm, 120, spots, False) + [_bermudan(rng, "rate") for _ in range(n_berm)]
        trades = [trades[i] for i in rng.permutation(len(trades))]
        books = _sets(rng, case, trades, True)
        csa = [gpu.compile(m, b, S.Options(pfe_quantile=PFE)) for b in books]
        grid = tuple(float(t) for t in csa[0].times)  # the plain twins on the margin-call dates too: one scenario
        plain = [gpu.compile(m, S.NettingSet(b.trades, None), S.Options(pfe_quantile=PFE, extra_dates=grid)) for b in books]
        return csa + plain
    m = _model(rng, case, case["months"], False)
    trades = _trades(rng, case["trades"], case["months"], [a.spot for a in m.assets], False)
    o = S.Options(pfe_quantile=PFE, im_quantile=0.99, im_inner_paths=case["inner"], im_margin_period=MPR)
    return [gpu.compile(m, S.NettingSet(trades, _csa(rng)), o)]


def _rows(case, seed):
    """Surrogate inputs and targets with the spreads of the book's features, and a starting network."""
    rng = np.random.default_rng([seed, 16])
    n = case["rows"]
    sd = np.array([0.02, 0.1, 0.1, 0.01, 1.0, 3.0, 0.5, 1, 1, 1, 0.03, 5.0, 0.2, 1.0, 0.1, 1.0], np.float32)
    z = rng.standard_normal((n, 16)).astype(np.float32)
    x = z * sd + np.arange(16, dtype=np.float32) * 0.1
    y = np.sin(z[:, 0]) + 0.5 * z[:, 1] * z[:, 2] + np.tanh(z[:, 4] - z[:, 5]) + 0.1 * z[:, 11] ** 2
    p = []
    for fan_in, out in ((16, 128), (128, 128), (128, 128), (128, 1)):
        a = math.sqrt(6.0 / fan_in)
        p += [rng.uniform(-a, a, fan_in * out), rng.uniform(-0.1, 0.1, out)]
    scaling = np.concatenate([x.mean(0), 1.0 / x.std(0), [y.mean(), y.std()]])
    return x, y.astype(np.float32), np.concatenate(p).astype(np.float32), scaling.astype(np.float32)


# ---------------------------------------------------------------------------------------------------------------
# One pass

_context = []


def _ctx():
    """The program's one context on the GPU."""
    if not _context:
        _context.append(gpu.Context(0))
    return _context[0]


def _fit(ctx, plans):
    return [ctx.fit_amc(p) if p.amc_degrees else p for p in plans]


def prepare(case, seed):
    if case["kind"] == "net":
        x, y, p, scaling = _rows(case, seed)
        net = Surrogate(_ctx(), seed=1)
        net.set_params(p, scaling)
        return {"case": case, "x": x, "y": y, "net": net}
    plans = _plans(case, seed)
    state = {"case": case, "plans": plans}
    if case["kind"] == "mixed":  # fitted and uploaded once, then revalued
        plans = _fit(_ctx(), plans[:case["sets"]])
        twins = [_like(f, p) for f, p in zip(plans, state["plans"][case["sets"]:])]
        state["batch"] = _ctx().batch(plans + twins)
    elif case.get("call") == "batch":
        state["batch"] = _ctx().batch(plans)
    else:
        _ctx()
    return state


def _like(fitted, plain):
    """The uncollateralised twin with the fitted records of the CSA plan (the same trades on the same dates)."""
    if fitted.amc_degrees and fitted.terms.shape == plain.terms.shape:
        plain.terms[:] = fitted.terms
    return plain


def _stacked(bufs):
    return {"sums": np.stack([s for s, _ in bufs]), "values": np.stack([v for _, v in bufs])}


def _outputs(state, bufs):
    n = state["case"]["sets"]
    return {"csa": _stacked(bufs[:n]), "plain": _stacked(bufs[n:])} if state["case"]["kind"] == "mixed" else _stacked(bufs)


def run(state):
    case, ctx = state["case"], _ctx()
    if case["kind"] == "net":
        if case["call"] == "gradients":
            loss, g = state["net"].gradients(state["x"], state["y"])
            return {"loss": np.array([loss], np.float32), "grad": g}
        return state["net"].predict(state["x"])
    if "batch" in state:
        state["batch"].execute()
        return _outputs(state, state["batch"].read())
    plans = state["plans"]
    if case["kind"] == "amc":
        fitted = _fit(ctx, plans)
        return [p.terms for p in fitted] if case["call"] == "fit" else _stacked(ctx.run_many(fitted))
    if case.get("call") == "f64":
        sums, values = ctx.run_f64(plans[0])
        return {"sums": sums, "values": values}
    return _stacked(ctx.run_many(plans) if len(plans) > 1 else [ctx.run(plans[0])])


def work(case):
    """Bytes: plan tables (or rows) in, statistics out.  Operations: per path, date and trade alive there about four
    cash flows of an exponential and two operations each (ten counted), and a path's step of its factors."""
    if case["kind"] == "net":
        params = 16 * 128 + 2 * 128 * 128 + 128
        n = case["rows"]
        back = case["call"] == "gradients"
        return {"bytes": n * (64 + 4) + 35_329 * (8 if back else 4), "flops": 2.0 * n * params * (3 if back else 1)}
    paths, months = case["paths"], case.get("months", 120)
    plans, dates, trades = case.get("sets", 1), 2 * months + 1, case.get("trades", 0)
    if case["kind"] == "amc":
        dates, trades = 41, 4 * case["bermudans"]
    elif case["kind"] == "mixed":
        plans, trades = 2 * plans, 2 * trades
    elif case["kind"] == "book" and not case["csa"]:
        dates = months + 1
    flops = paths * dates * (200.0 + 0.5 * trades * 4 * 10)
    if case["kind"] == "margin":
        flops += paths * (months + 1) * case["inner"] * (100.0 + 0.5 * trades * 4 * 10)
    if case["kind"] == "amc" and case["call"] == "fit":
        out = plans * 41 * 32.0
    else:
        out = plans * dates * 8 * 4.0
    return {"bytes": 32.0 * dates * 0.5 * trades * 4 + out, "flops": flops}


# ---------------------------------------------------------------------------------------------------------------
# The same in 64 bits

F64 = torch.float64
M32 = 0xFFFFFFFF


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _pcg(v):
    state = (v * 747796405 + 2891336453) & M32
    word = (((state >> ((state >> 28) + 4)) ^ state) * 277803737) & M32
    return (word >> 22) ^ word


def _pcg_int(v):
    return int(_pcg(torch.tensor(v, dtype=torch.int64)))


class _Scenario:
    """The simulated factors of a plan, date by date: x, D, S[a], Q[c], xf[f], each [paths]."""

    def __init__(self, header, params, steps, dev):
        h = [int(v) for v in header]
        self.P, self.T, self.nA, self.nC, self.sub, self.nN, self.seed, self.anti = h[:8]
        self.cpty, self.nCorr = h[9], h[11]
        self.nF = (h[10] - 6) // 2
        self.steps = np.asarray(steps, np.float64).reshape(self.T, 4 * h[10])
        self.prm = np.asarray(params, np.float64)
        self.chol = torch.tensor(self.prm[16:80].reshape(8, 8), device=dev)
        path = torch.arange(self.P, dtype=torch.int64, device=dev)
        stream = path >> 1 if self.anti else path
        self.sign = (1.0 - 2.0 * (path & 1).to(F64)) if self.anti else torch.ones(self.P, dtype=F64, device=dev)
        self.stream = _pcg(_pcg_int(self.seed) ^ _pcg((stream + 0x9E3779B9) & M32))
        zero = torch.zeros(self.P, dtype=F64, device=dev)
        self.x, self.lnD, self.D = zero, zero, zero + 1.0
        self.lnS = [zero] * self.nA
        self.S = [zero + self.prm[12 + a] for a in range(self.nA)]
        self.xf = [zero] * self.nF
        self.y, self.Y = [zero + self.prm[4 * c + 3] for c in range(self.nC)], [zero] * self.nC
        self.Q = [zero + 1.0] * self.nC

    def step(self, j):
        if j == 0:
            return
        z = []
        for q in range((self.nN + 1) // 2):
            h1 = _pcg(self.stream ^ _pcg_int(j * 131 + q))
            h2 = _pcg(h1 ^ 0x68E31DA4)
            u1, u2 = ((h1 >> 8).to(F64) + 0.5) / 16777216.0, ((h2 >> 8).to(F64) + 0.5) / 16777216.0
            r, a = torch.sqrt(-2.0 * torch.log(u1)), (2.0 * math.pi) * u2
            z += [self.sign * r * torch.cos(a), self.sign * r * torch.sin(a)]
        w = self.chol[:, :self.nCorr] @ torch.stack(z[:self.nCorr])
        st, nCorr = self.steps[j], self.nCorr
        integrated = self.x * st[5] + st[2] * w[0] + st[3] * z[nCorr] + st[4]
        self.x = self.x * st[0] + st[1] * w[0]
        self.lnD = self.lnD - integrated
        self.D = torch.exp(self.lnD)
        carry = [st[8 + a] for a in range(4)]
        for f in range(self.nF):
            fs = st[24 + 8 * f:32 + 8 * f]
            wf = w[1 + self.nA + self.nC + f]
            carry[f] = self.xf[f] * fs[5] + fs[2] * wf + fs[3] * z[nCorr + 1 + f] + fs[4] + fs[7]
            self.xf[f] = self.xf[f] * fs[0] + fs[1] * wf + fs[6]
        for a in range(self.nA):
            self.lnS[a] = self.lnS[a] + (integrated - carry[a] - st[16 + a] + st[12 + a] * w[1 + a])
            self.S[a] = self.prm[12 + a] * torch.exp(self.lnS[a])
        off = nCorr + 1 + self.nF
        for c in range(self.nC):
            kappa, theta, xi = self.prm[4 * c:4 * c + 3]
            dt = st[6]
            h, rem, left = dt / self.sub, math.sqrt(dt) * w[1 + self.nA + c], dt
            for s in range(self.sub):
                dW = rem
                if s + 1 < self.sub:
                    dW = (h / left) * rem + math.sqrt(max(h * (left - h) / left, 0.0)) * z[off + s]
                rem, left = rem - dW, left - h
                yp = self.y[c].clamp(min=0.0)
                yn = self.y[c] + kappa * (theta - yp) * h + xi * torch.sqrt(yp) * dW
                self.Y[c] = self.Y[c] + 0.5 * (yp + yn.clamp(min=0.0)) * h
                self.y[c] = yn
            off += self.sub - 1
            self.Q[c] = torch.exp(-self.Y[c] - st[20 + c])


def _black(F, K, sd, df, call):
    s = torch.where(call, 1.0, -1.0).to(F64)[:, None]
    K, sd = K[:, None], sd[:, None]
    flat = sd <= 1e-7
    sd = torch.where(flat, torch.ones_like(sd), sd)
    d1 = torch.log(F / K) / sd + 0.5 * sd
    cdf = lambda v: 0.5 * torch.erfc(-v / math.sqrt(2.0))  # noqa: E731
    price = df * s * (F * cdf(s * d1) - K * cdf(s * (d1 - sd)))
    return torch.where(flat, df * (s * (F - K)).clamp(min=0.0), price)


def _monomials(z, w=None):
    if w is None:
        return torch.stack([torch.ones_like(z), z, z * z, z * z * z], 1)
    return torch.stack([torch.ones_like(z), z, w, z * z, z * w, w * w, z ** 3, z * z * w, z * w * w, w ** 3], 1)


class _Fit:
    """One regression of y on the standardised state (and swap rate) at degree 3, by its ridged normal equations."""

    def __init__(self, x, y, s=None):
        self.cx, self.sx = x.mean(), x.std(unbiased=False)
        self.cs = self.ss = None
        if s is not None:
            self.cs, self.ss = s.mean(), s.std(unbiased=False)
        if float(self.sx) < 1e-12:  # today's state: the mean
            self.c = torch.zeros(4 if s is None else 10, dtype=F64, device=x.device)
            self.c[0] = y.mean()
            self.sx = torch.ones_like(self.sx)
            if s is not None:
                self.cx, self.cs, self.ss = 0 * self.cx, 0 * self.cs, torch.ones_like(self.ss)
            return
        A = self.design(x, s)
        G = A.T @ A
        G.diagonal().add_((1e-12 if s is None else 1e-6) * x.numel())
        self.c = torch.linalg.solve(G, A.T @ y)

    def design(self, x, s):
        return _monomials((x - self.cx) / self.sx, None if s is None else (s - self.cs) / self.ss)

    def __call__(self, x, s=None):
        return self.design(x, s) @ self.c


def _bermudans(plans, tables, scenario):
    """The fits of every Bermudan of the plans: {(plan, term): _Fit} for policy and continuation terms, and the fitted
    records written into a copy of each term table."""
    dev = _device()
    recs = []  # (plan, Bermudan, date, term, kind, exercise index)
    value = {}
    X, D = [], []
    sc = scenario()
    many = [len(p.amc_degrees) > 4 for p in plans]
    swap = {}
    for j in range(sc.T):
        sc.step(j)
        X.append(sc.x), D.append(sc.D)
        for i, (p, t) in enumerate(zip(plans, tables)):
            ann = flt = 0.0
            for u in range(int(p.indices[j]), int(p.indices[j + 1])):
                r = t[u]
                code = int(r[0])
                kind = code & 15
                if kind < 5 or kind == 10:
                    continue
                b = ((code >> 8) & 15) | (((code >> 4) & 15) << 4 if many[i] else 0)
                bond = r[2] * r[3] * torch.exp(-r[4] * sc.x) if kind in (5, 13, 14) else None
                if kind == 5:
                    value[i, b, j] = value.get((i, b, j), 0.0) + bond
                elif kind == 13:
                    ann = ann + bond
                elif kind == 14:
                    flt = flt + bond
                elif kind in (6, 7):
                    if isinstance(ann, torch.Tensor):
                        swap[i, u] = flt / ann
                    ann = flt = 0.0
                    recs.append((i, b, j, u, kind, code >> 12))
    fits = {}
    for i, p in enumerate(plans):
        for b in range(len(p.amc_degrees)):
            mine = [r for r in recs if r[0] == i and r[1] == b]
            policy = sorted((r for r in mine if r[4] == 6), key=lambda r: r[5])
            realised = torch.zeros(sc.P, dtype=F64, device=dev)
            for k in range(len(policy) - 1, -1, -1):
                _, _, j, u, _, _ = policy[k]
                e = value[i, b, j]
                itm = e > 0.0
                s = swap.get((i, u))
                f = _Fit(X[j][itm], (realised / D[j])[itm], None if s is None else s[itm])
                fits[i, u] = f
                take = itm & (e > f(X[j], s))
                realised = torch.where(take, D[j] * e, realised)
                first = policy[k - 1][2] if k else 0
                for _, _, jc, uc, kind, _ in mine:
                    if kind == 7 and first <= jc < j:
                        fits[i, uc] = _Fit(X[jc], realised / D[jc], swap.get((i, uc)))
    out = []
    for i, t in enumerate(tables):
        t = t.copy()
        for (k, u), f in fits.items():
            if k != i:
                continue
            c = [float(v) for v in f.c]
            if f.cs is None:
                t[u, 2:8] = [float(f.cx), 1.0 / float(f.sx)] + c
            else:
                t[u, 2:8] = [float(f.cx), 1.0 / float(f.sx), float(f.cs), 1.0 / float(f.ss)] + c[:2]
                t[u + 1, 1:8], t[u + 2, 1] = c[2:9], c[9]
        out.append(t)
    return fits, out


def _statistics(plans, f64):
    """sums and values of plans that share a scenario, as the fused pipeline defines them."""
    dev = _device()
    p0 = plans[0]
    if f64:
        params = [p.tables64["params"] for p in plans]
        tables = [np.asarray(p.tables64["terms"], np.float64).reshape(-1, 8) for p in plans]
        steps = p0.tables64["steps"]
        requests = [np.asarray(p.tables64["requests"], np.float64).reshape(-1, 8) for p in plans]
    else:
        params = [np.asarray(p.params, np.float64) for p in plans]
        tables = [p.terms.astype(np.float64).reshape(-1, 8) for p in plans]
        steps = p0.steps
        requests = [p.requests.astype(np.float64).reshape(-1, 8) for p in plans]

    def scenario():
        return _Scenario(p0.header, params[0], steps, dev)

    fits = _bermudans(plans, tables, scenario)[0] if any(p.amc_degrees for p in plans) else {}
    sc = scenario()
    n, P, T = len(plans), sc.P, sc.T
    many = [len(p.amc_degrees) > 4 for p in plans]
    fix = torch.zeros((n, 32, P), dtype=F64, device=dev)
    exercised = {}  # (plan, Bermudan): the exercise index of each path, -1 before
    prm = torch.tensor(np.stack(params), device=dev)
    csa = torch.tensor([bool(p.header[8]) for p in plans], device=dev)[:, None]
    hc, hb, mta, ia = (prm[:, 8 + k][:, None] for k in range(4))
    hb = torch.where(hb >= 0.0, hb, torch.full_like(hb, math.inf))
    held = torch.zeros((n, P), dtype=F64, device=dev)
    prev_de, prev_q = torch.zeros((n, P), dtype=F64, device=dev), torch.ones(P, dtype=F64, device=dev)
    past = {}
    sums = torch.zeros((n, T, 8), dtype=F64, device=dev)
    values = np.full((n, max(1, p0.num_outputs)), np.nan)
    wanted = {}  # row: [(plan, output, level)] of the quantile requests
    for i, rq in enumerate(requests):
        for r in rq:
            if int(r[0]) == 0:
                wanted.setdefault(int(r[1]), []).append((i, int(r[7]), float(r[4])))
    spans = [np.diff(p.indices[:T + 1].astype(np.int64)) for p in plans]
    t64 = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=F64, device=dev)  # noqa: E731
    for j in range(T):
        sc.step(j)
        rec = np.concatenate([t[int(p.indices[j]):int(p.indices[j + 1])] for p, t in zip(plans, tables)])
        of = np.repeat(np.arange(n), [int(s[j]) for s in spans])
        at = np.concatenate([np.arange(int(p.indices[j]), int(p.indices[j + 1])) for p in plans])
        code = rec[:, 0].astype(np.int64)
        kind, extra = code & 15, code >> 12
        value = torch.zeros((n, P), dtype=F64, device=dev)
        # every bond, and the fixed part of every running coupon: distinct exponents once, then one product
        sel = np.nonzero((kind == 0) | (kind == 1))[0]
        if len(sel):
            B, which = np.unique(rec[sel, 4], return_inverse=True)
            amount = np.where(kind[sel] == 0, rec[sel, 2], rec[sel, 5]) * rec[sel, 3]
            coef = np.zeros((n, len(B)))
            np.add.at(coef, (of[sel], which), amount)
            value += t64(coef) @ torch.exp(-t64(B)[:, None] * sc.x)
        sel = np.nonzero(kind == 1)[0]
        for a in range(0, len(sel), 64):
            q = sel[a:a + 64]
            E = torch.exp(-t64(rec[q, 4])[:, None] * sc.x) * t64(rec[q, 2] * rec[q, 3])[:, None]
            value.index_add_(0, torch.tensor(of[q], device=dev), E * fix[of[q], rec[q, 1].astype(np.int64)])
        for q in np.nonzero(kind == 2)[0]:
            value[of[q]] += rec[q, 2] * rec[q, 3] * sc.S[int(rec[q, 1]) & 3]
        for q in np.nonzero(kind == 11)[0]:
            a = int(extra[q])
            value[of[q]] += rec[q, 2] * rec[q, 3] * sc.S[a] * torch.exp(-rec[q, 1] * sc.xf[a])
        sel = np.nonzero((kind == 4) | (kind == 12))[0]
        for a in range(0, len(sel), 64):
            q = sel[a:a + 64]
            asset = [int(extra[k]) if kind[k] == 12 else int(rec[k, 1]) & 3 for k in q]
            fwd = torch.stack([sc.S[s] * (torch.exp(-rec[k, 1] * sc.xf[s]) if kind[k] == 12 else 1.0) for k, s in zip(q, asset)])
            b0 = t64(rec[q, 3])[:, None] * torch.exp(-t64(rec[q, 4])[:, None] * sc.x)
            v = _black(fwd * t64(rec[q, 5])[:, None] / b0, t64(rec[q, 6]), t64(np.abs(rec[q, 7])), b0,
                       torch.tensor(rec[q, 7] > 0.0, device=dev))
            value.index_add_(0, torch.tensor(of[q], device=dev), v * t64(rec[q, 2])[:, None])
        ev, ann, flt = {}, {}, {}
        for q in np.nonzero((kind >= 5) & (kind != 10) & (kind != 11) & (kind != 12))[0]:  # Bermudans, in plan order
            i, k, r = int(of[q]), int(kind[q]), rec[q]
            if k == 15:
                continue
            b = ((int(code[q]) >> 8) & 15) | (((int(code[q]) >> 4) & 15) << 4 if many[i] else 0)
            ex = exercised.setdefault((i, b), torch.full((P,), -1, dtype=torch.int64, device=dev))
            if k in (6, 7):
                f, s = fits[i, int(at[q])], None
                if i in ann:
                    s = flt.pop(i) / ann.pop(i)
                cont = f(sc.x, s)
                if k == 6:
                    e = ev[i, b]
                    exercised[i, b] = torch.where((ex < 0) & (e > 0.0) & (e > cont), int(extra[q]), ex)
                else:
                    value[i] += torch.where(ex < 0, r[1] * cont.clamp(min=0.0), 0.0)
                continue
            bond = r[3] * torch.exp(-r[4] * sc.x)
            if k == 5:
                ev[i, b] = ev.get((i, b), 0.0) + r[2] * bond
            elif k == 13:
                ann[i] = ann.get(i, 0.0) + r[2] * bond
            elif k == 14:
                flt[i] = flt.get(i, 0.0) + r[2] * bond
            else:
                live = (ex >= 0) & (ex <= int(extra[q]))
                amount = r[2] if k == 8 else r[2] * fix[i, int(r[1])] + r[5]
                value[i] += torch.where(live, amount * bond, 0.0)
        sel = np.nonzero(kind == 3)[0]
        for a in range(0, len(sel), 64):  # after every use of the previous fixing
            q = sel[a:a + 64]
            E = torch.exp(-t64(rec[q, 4])[:, None] * sc.x) * t64(rec[q, 3])[:, None]
            fix[of[q], rec[q, 1].astype(np.int64)] = (E - 1.0) / t64(rec[q, 2])[:, None]
        # cash collateral called on the value at the call date
        past[j] = value
        call = [int(p.indices[T + 1 + j]) for p in plans]
        vc = past[call[0]] if len(set(call)) == 1 else torch.stack([past[c][i] for i, c in enumerate(call)])
        past = {k: v for k, v in past.items() if k >= j - 4}
        required = (vc - hc).clamp(min=0.0) + (vc + hb).clamp(max=0.0)
        held = torch.where(((required - held).abs() >= mta) | (j == 0), required, held)
        e = value - torch.where(csa, held + ia, 0.0)
        ep, en = e.clamp(min=0.0), e.clamp(max=0.0)
        Q = sc.Q[sc.cpty] if sc.nC else torch.ones(P, dtype=F64, device=dev)
        slots = [int(p.indices[2 * T + 1 + j]) for p in plans]
        inc = torch.zeros((n, P), dtype=F64, device=dev)
        if slots[0] > 0:
            de = sc.D * ep
            if j > 0:
                inc = 0.5 * (prev_de + de) * (prev_q - Q)
            prev_de, prev_q = de, Q
            for i, p in enumerate(plans):
                for who, out, level in wanted.get(int(p.header[28]) + slots[i] - 1, []):
                    if who == i:
                        h = level * (P - 1)
                        k = min(int(h), P - 1)
                        v = torch.sort(ep[i]).values
                        values[i, out] = float(v[k] + (h - k) * (v[min(k + 1, P - 1)] - v[k]))
        for k, v in enumerate((e, ep, en, sc.D * ep, sc.D * en, inc)):
            sums[:, j, k] = v.mean(1)
        sums[:, j, 6], sums[:, j, 7] = Q.mean(), sc.D.mean()
    return sums.reshape(n, T * 8).cpu().numpy(), values


def _network(case, seed):
    dev = _device()
    x, y, p, scaling = _rows(case, seed)
    sc = torch.tensor(scaling.astype(np.float64), device=dev)
    w, o = [], 0
    for shape in ((128, 16), (128,), (128, 128), (128,), (128, 128), (128,), (1, 128), (1,)):
        k = int(np.prod(shape))
        w.append(torch.tensor(p[o:o + k].astype(np.float64).reshape(shape), device=dev, requires_grad=True))
        o += k
    h = (torch.tensor(x, device=dev).to(F64) - sc[:16]) * sc[16:32]
    for k in range(3):
        h = torch.nn.functional.silu(h @ w[2 * k].T + w[2 * k + 1])
    out = (h @ w[6].T + w[7])[:, 0]
    if case["call"] == "predict":
        return (out * sc[33] + sc[32]).detach().cpu().numpy()
    loss = ((out - (torch.tensor(y, device=dev).to(F64) - sc[32]) / sc[33]) ** 2).mean()
    loss.backward()
    return {"loss": np.array([float(loss)]), "grad": torch.cat([v.grad.reshape(-1) for v in w]).cpu().numpy()}


def exact(case, seed):
    if case["kind"] == "net":
        return _network(case, seed)
    # The dates' values of every netting set on every path are formed at once: what does not fit is left out.
    if case["kind"] == "mixed" or case["paths"] * case.get("sets", 1) > 12_000_000:
        return None
    plans = _plans(case, seed)
    if case["kind"] == "amc" and case["call"] == "fit":
        tables = [p.terms.astype(np.float64).reshape(-1, 8) for p in plans]
        p0 = plans[0]
        fitted = _bermudans(plans, tables, lambda: _Scenario(p0.header, p0.params, p0.steps, _device()))[1]
        return [t.reshape(-1) for t in fitted]
    sums, values = _statistics(plans, case.get("call") == "f64")
    if case["kind"] == "margin":  # the inner simulation is not restated
        return {"sums": sums, "values": None}
    return {"sums": sums[0], "values": values[0]} if case.get("call") == "f64" else {"sums": sums, "values": values}
