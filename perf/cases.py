"""Performance cases of the engine, through the entry points that a program calls.

Each case is one synchronous call of ``compfinance_gb300.Engine`` (or, for ``serve``, one batch of
requests through ``compfinance_gb300.Server``) on a stored model and product, as a pricing or risk
program makes it again and again.  Sizes are those of the repository's workloads: the
Black-Scholes European, the Dupire barrier on 20x10, 60x30 and 120x60 grids with 12 to 520 steps,
the 200-option portfolio and its superbucket, the four-asset autocall and basket, and the mixed
serving stream.  Surfaces, spots and generator seeds are made from the case's seed.

``exact`` restates the mathematics in 64-bit torch: the generators are whole-number recurrences,
the inverse normal and the log-Euler step are the reference's formulas, risks are path-wise
adjoints.
"""
import math
import os
import random

import numpy as np
import torch

from compfinance_gb300 import Engine, NumericalParam
from compfinance_gb300.api import Server
from compfinance_gb300 import workloads as W

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MONTH = 1.0 / 12.0


def listed():
    """The cases; the comment above each says what it stands for."""
    return [
        # the smallest call: the serving stream's most frequent request, one Black-Scholes value
        dict(name="bs_value", kind="bs_value", paths=1 << 14, sobol=True, precision="fp32"),
        # price and four Greeks of a European, the plain method in double precision
        dict(name="bs_risk", kind="bs_risk", paths=1 << 16, sobol=True, precision="fp64"),
        # price only of the weekly barrier, default precision
        dict(name="uoc_value", kind="uoc_value", nS=60, nT=30, steps=156, paths=1 << 18, sobol=False, precision="fp64"),
        # price and all 1801 risks of the weekly barrier, default precision
        dict(name="uoc_risk", kind="uoc_risk", nS=60, nT=30, steps=156, paths=1 << 18, sobol=False, precision="fp64",
             update=False),
        # the largest: the same risk at production path count in the FP32-path form, the market
        # data stored anew before every run
        dict(name="uoc_risk_fp32", kind="uoc_risk", nS=60, nT=30, steps=156, paths=1 << 22, sobol=False,
             precision="fp32", update=True),
        # a fine grid with many steps and an odd number of paths
        dict(name="uoc_risk_fine_fp32", kind="uoc_risk", nS=120, nT=60, steps=520, paths=200_001, sobol=False,
             precision="fp32", update=False),
        # mcSimul: every path's payoffs of a barrier on a coarse grid, an odd number of paths
        dict(name="uoc_paths", kind="uoc_paths", nS=20, nT=10, steps=52, paths=100_001, sobol=False, precision="fp64"),
        # risk of each of 200 options (AADriskMulti) at the serving stream's path count
        dict(name="multi_fp32", kind="multi", nS=60, nT=30, payoffs=200, paths=1 << 16, sobol=True, precision="fp32"),
        # the same in double precision
        dict(name="multi", kind="multi", nS=60, nT=30, payoffs=200, paths=1 << 18, sobol=True, precision="fp64"),
        # implied-vol risk of the 200-option book: calibration, Monte Carlo adjoints, calibration
        # adjoint; FP32-path form (the calibration divides a second difference by 1e-8, so its
        # vegas have no 64-bit value that another evaluation order would reproduce)
        dict(name="superbucket_fp32", kind="superbucket", payoffs=200, paths=1 << 20, sobol=True, precision="fp32"),
        # four correlated assets: price and 36 risks of the autocall, default precision
        dict(name="autocall_risk", kind="autocall", paths=1 << 18, sobol=True, precision="fp64"),
        # a batch of the mixed serving stream, all in flight together
        dict(name="serve", kind="serve", requests=24, mix=7, precision="fp32"),
    ]


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["bs_value", "bs_risk", "uoc_value", "uoc_risk", "uoc_risk", "uoc_paths", "multi", "superbucket",
                       "autocall", "basket", "serve"])

    def paths(lo, hi):
        n = int(round(2.0 ** rng.uniform(math.log2(lo), math.log2(hi))))
        return n if rng.random() < 0.5 else max(32, n // 256 * 256)

    precision = rng.choice(["fp64", "fp32"])
    sobol = rng.random() < 0.5
    c = dict(kind=kind, precision=precision)
    if kind in ("bs_value", "bs_risk"):
        return dict(c, paths=paths(1 << 12, 1 << 20), sobol=sobol)
    if kind in ("uoc_value", "uoc_risk", "uoc_paths"):
        nS, nT = rng.choice([(20, 10), (60, 30), (120, 60)])
        steps = rng.choice([12, 52, 156, 520])
        # at most about 4e7 path-steps in double precision and 6e8 in the FP32-path form
        top = min(1 << 22, (4 << 23 if precision == "fp64" else 6 << 26) // steps)
        if kind == "uoc_paths":
            top = min(top, 1 << 19)
        c.update(nS=nS, nT=nT, steps=steps, paths=paths(1 << 14, top), sobol=sobol)
        if kind == "uoc_risk":
            c["update"] = rng.random() < 0.3
        return c
    if kind == "multi":
        nS, nT = rng.choice([(20, 10), (60, 30), (120, 60)])
        return dict(c, nS=nS, nT=nT, payoffs=rng.choice([50, 100, 150, 200]),
                    paths=paths(1 << 14, 1 << 18 if precision == "fp64" else 1 << 20), sobol=True)
    if kind == "superbucket":
        return dict(c, precision="fp32", payoffs=rng.choice([50, 100, 200]), paths=paths(1 << 15, 1 << 20), sobol=True)
    if kind in ("autocall", "basket"):
        return dict(c, paths=paths(1 << 14, 1 << 18 if precision == "fp64" else 1 << 20), sobol=sobol)
    return dict(c, precision="fp32", requests=rng.randint(8, 24), mix=rng.randint(0, 10_000))


# ---------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------
_shared = {}


def _engine():
    """The program's one context on the GPU."""
    if "eng" not in _shared:
        _shared["eng"] = Engine(0)
    return _shared["eng"]


def _server():
    """The program's one server: lanes and admission order as the serving benchmark runs it."""
    if "srv" not in _shared:
        srv = Server(_engine(), slots=11, hbm_budget=64 << 30)
        srv.configure(short_slots=8, long_threshold=2e7, long_blocks_per_sm=4)
        srv.order(1, 1, 50.0)
        _shared["srv"] = srv
    return _shared["srv"]


def _surface(nS, nT, rs):
    """Local vols on log-spaced spots over 50-200 and times over 0.1-3: smile plus seeded noise."""
    spots = 50.0 * 4.0 ** (np.arange(nS) / (nS - 1))
    times = 0.1 + 2.9 * np.arange(nT) / (nT - 1)
    v = 0.15 + 0.10 * np.exp(-times)[None, :] * np.log(spots / 100.0)[:, None] ** 2
    return spots, times, np.maximum(0.05, v + 0.005 * rs.standard_normal((nS, nT)))


def _dupire(case, rs, max_dt):
    spots, times, vols = _surface(case["nS"], case["nT"], rs)
    return dict(spot=round(rs.uniform(95.0, 105.0), 2), spots=spots, times=times, vols=vols, max_dt=max_dt)


def _barrier(steps, strike=120.0, barrier=150.0):
    return dict(strike=strike, barrier=barrier, maturity=3.0, freq=3.0 / steps, smooth=0.01)


def _portfolio(payoffs, spot=100.0):
    """10 maturities over 0.3-3y, strikes 0.7-1.6 of the spot."""
    nk = payoffs // 10
    mats = [0.3 + 2.7 * j / 9 for j in range(10) for _ in range(nk)]
    strikes = [spot * (0.7 + 0.9 * i / max(1, nk - 1)) for _ in range(10) for i in range(nk)]
    return mats, strikes


def _requests(case):
    """The batch's requests in arrival order, in the stream's proportions and sizes."""
    r, out = random.Random(case["mix"]), []
    for i in range(case["requests"]):
        u = (i * 10 // case["requests"]) / 10
        grid, strike, bar = r.choice(W.SERVE_GRIDS), r.choice(W.SERVE_KR_BARRIER), r.choice(W.SERVE_BR)
        if u < 0.4:
            out.append(dict(kind="value", strike=100.0 * r.choice(W.SERVE_KR), paths=1 << 14, sobol=True))
        elif u < 0.8:
            out.append(dict(kind="risk", grid=grid, strike=100.0 * strike, barrier=100.0 * bar,
                            steps=r.choice(W.SERVE_STEPS), paths=int(round(2.0 ** r.uniform(16, 20) / 256)) * 256,
                            sobol=False))
        else:
            out.append(dict(kind="multi", grid=grid, payoffs=r.choice(W.SERVE_NPAY), paths=1 << 16, sobol=True))
    r.shuffle(out)
    return out


def _inputs(case, seed):
    """What the case runs on, as plain numbers and arrays."""
    rs = np.random.RandomState((seed * 7919 + 17) % (1 << 32))
    kind = case["kind"]
    d = dict(seed1=int(rs.randint(1, 1 << 30)), seed2=int(rs.randint(1, 1 << 30)))
    if kind in ("bs_value", "bs_risk"):
        d["bs"] = dict(spot=round(rs.uniform(95, 105), 2), vol=round(rs.uniform(0.15, 0.25), 4), rate=0.02, div=0.0)
        d["strike"], d["maturity"] = 100.0, 1.0
    elif kind in ("uoc_value", "uoc_risk", "uoc_paths"):
        d["model"], d["uoc"] = _dupire(case, rs, 0.25), _barrier(case["steps"])
    elif kind == "multi":
        d["model"], d["portfolio"] = _dupire(case, rs, MONTH), _portfolio(case["payoffs"])
    elif kind == "superbucket":
        d["ivs"] = [W.SB_IVS["a"] + 0.01 * rs.uniform(), W.SB_IVS["b"], W.SB_IVS["c"], W.SB_IVS["sref"]]
        d["portfolio"] = _portfolio(case["payoffs"])
        d["notionals"] = rs.uniform(0.5, 1.5, case["payoffs"])
    elif kind in ("autocall", "basket"):
        m = dict(W.MD4)
        m["spots"] = [s * rs.uniform(0.97, 1.03) for s in m["spots"]]
        # the last asset's vol keeps it at the normal dynamics (vol + 2 skew = 0)
        m["atms"] = [a * rs.uniform(0.95, 1.05) for a in m["atms"][:3]] + m["atms"][3:]
        d["md"] = m
    else:
        d["bs"] = dict(spot=100.0, vol=round(rs.uniform(0.15, 0.25), 4), rate=0.02, div=0.0)
        d["models"] = {g: _dupire(dict(nS=g[0], nT=g[1]), rs, 0.25) for g in W.SERVE_GRIDS}
        d["requests"] = _requests(case)
    return d


def _put_dupire(eng, m, mid, max_dt=None):
    return eng.putDupire(m["spot"], m["spots"], m["times"], m["vols"], max_dt or m["max_dt"], mid)


def _put_barrier(eng, u, pid):
    return eng.putBarrier(u["strike"], u["barrier"], u["maturity"], u["freq"], u["smooth"], False, pid)


def prepare(case, seed):
    eng, d, kind = _engine(), _inputs(case, seed), case["kind"]
    tag = "%s_%d" % (kind, seed)
    s = dict(eng=eng, kind=kind, mid=tag + "_m", pid=tag + "_p")
    if kind != "serve":
        s["num"] = NumericalParam(useSobol=case["sobol"], numPath=case["paths"], seed1=d["seed1"], seed2=d["seed2"],
                                  precision=case["precision"])
    if "bs" in d and kind != "serve":
        b = d["bs"]
        eng.putBlackScholes(b["spot"], b["vol"], False, b["rate"], b["div"], s["mid"])
        eng.putEuropean(d["strike"], d["maturity"], id=s["pid"])
    elif "uoc" in d:
        _put_dupire(eng, d["model"], s["mid"])
        _put_barrier(eng, d["uoc"], s["pid"])
        s["update"] = d["model"] if case.get("update") else None
    elif kind == "multi":
        _put_dupire(eng, d["model"], s["mid"])
        eng.putEuropeans(*d["portfolio"], s["pid"])
    elif kind == "superbucket":
        eng.putEuropeans(*d["portfolio"], s["pid"])
        s["args"] = (Engine.ivs("param", 100.0, d["ivs"]), 100.0, MONTH, s["pid"], d["notionals"],
                     *W.superbucket_grid(60, 30), *W.superbucket_riskview(30, 12), s["num"])
    elif kind in ("autocall", "basket"):
        m, a, b = d["md"], W.MD4_AUTOCALL, W.MD4_BASKET
        eng.putDisplaced(m["assets"], m["spots"], m["atms"], m["skews"], m["disc"], m["spreads"], m["div_dates"],
                         m["divs"], m["correl"], m["lam"], s["mid"])
        if kind == "autocall":
            eng.putAutocall(m["assets"], a["refs"], a["maturity"], a["periods"], a["ko"], a["strike"], a["cpn"],
                            a["smooth"], s["pid"])
        else:
            eng.putBaskets(m["assets"], b["weights"], b["maturity"], b["strikes"], s["pid"])
    else:
        s["srv"], s["requests"] = _server(), []
        b = d["bs"]
        eng.putBlackScholes(b["spot"], b["vol"], False, b["rate"], b["div"], tag + "_bs")
        for g, m in d["models"].items():
            _put_dupire(eng, m, "%s_%dw" % (tag, g[0]))
            _put_dupire(eng, m, "%s_%dm" % (tag, g[0]), MONTH)
        for i, r in enumerate(d["requests"]):
            pid = "%s_p%d" % (tag, i)
            if r["kind"] == "value":
                mid = tag + "_bs"
                eng.putEuropean(r["strike"], 1.0, id=pid)
            elif r["kind"] == "risk":
                mid = "%s_%dw" % (tag, r["grid"][0])
                _put_barrier(eng, _barrier(r["steps"], r["strike"], r["barrier"]), pid)
            else:
                mid = "%s_%dm" % (tag, r["grid"][0])
                eng.putEuropeans(*_portfolio(r["payoffs"]), pid)
            s["requests"].append((r["kind"], mid, pid, NumericalParam(
                useSobol=r["sobol"], numPath=r["paths"], seed1=d["seed1"], seed2=d["seed2"],
                precision=case["precision"])))
    return s


def run(s):
    eng, kind = s["eng"], s["kind"]
    if kind == "serve":
        srv = s["srv"]
        ids = [srv.submit(*r) for r in s["requests"]]
        values, stderrs, risks = [], [], []
        for rid, (what, _, _, _) in zip(ids, s["requests"]):
            if srv.wait(rid) != "done":
                raise RuntimeError(srv.error())
            r = srv.result(rid)
            values.append(r["values"])
            if what == "value":
                stderrs.append(r["stderrs"])
            else:
                risks.append(r["risks"].reshape(-1))
            srv.release(rid)
        return dict(values=np.concatenate(values), stderrs=np.concatenate(stderrs) if stderrs else np.zeros(0),
                    risks=np.concatenate(risks) if risks else np.zeros(0))
    if kind in ("bs_value", "uoc_value"):
        r = eng.value(s["mid"], s["pid"], s["num"])
        return dict(values=r["values"], stderrs=r["stderrs"])
    if kind == "uoc_paths":
        return eng.simulatePaths(s["mid"], s["pid"], s["num"])
    if kind == "multi":
        r = eng.AADriskMulti(s["mid"], s["pid"], s["num"])
        return dict(values=r["values"], risks=r["risks"])
    if kind == "superbucket":
        r = eng.dupireSuperbucket(*s["args"])
        return dict(value=r["value"], delta=r["delta"], vega=r["vega"], microbucket=r["microbucket"])
    if s.get("update") is not None:
        _put_dupire(eng, s["update"], s["mid"])
    r = eng.AADriskOne(s["mid"], s["pid"], s["num"])
    return dict(values=r["payoffValues"], value=r["riskPayoffValue"], risks=r["risks"])


def work(case):
    """Flops of one path-step counted from the reference's source: 8 for an mrg32k3a draw, 29 for
    the Gaussian and the step, 16 for its adjoint.  Bytes: market data in, results out."""
    kind = case["kind"]

    def one(kind, n, nS=0, nT=0, steps=1, payoffs=1):
        nodes, f = nS * nT, 0.0
        if kind in ("bs_value", "bs_risk"):
            return 8 * 12, n * (37.0 + 20.0 + (20.0 if kind == "bs_risk" else 0.0))
        if kind in ("uoc_value", "uoc_paths"):
            return 8 * (nodes + nS + nT) + 16 * (n if kind == "uoc_paths" else 2), 37.0 * n * steps
        if kind == "uoc_risk":
            return 8 * (nodes + nS + nT) + 8 * (nodes + 4), 53.0 * n * steps
        if kind == "multi":
            # one adjoint per maturity that a path is in the money for, half of them on average
            for e in range(1, 11):
                f += 0.5 * n * 16.0 * steps * e / 10
            return 8 * (nodes + nS + nT) + 8 * (nodes + 2) * payoffs, 29.0 * n * steps + f
        return 0, 0.0

    if kind == "serve":
        got = [one({"value": "bs_value", "risk": "uoc_risk", "multi": "multi"}[r["kind"]], r["paths"],
                   *r.get("grid", (0, 0)), steps=r.get("steps", 40), payoffs=r.get("payoffs", 1))
               for r in _requests(case)]
        return dict(bytes=sum(g[0] for g in got), flops=sum(g[1] for g in got))
    if kind == "superbucket":
        b, f = one("multi", case["paths"], 60, 30, 40, 1)
        return dict(bytes=b + 8 * 360, flops=f + 60 * 30 * 5 * 200.0)
    if kind in ("autocall", "basket"):
        steps = W.MD4_AUTOCALL["periods"] if kind == "autocall" else 1
        return dict(bytes=8 * 36 * 2, flops=case["paths"] * steps * 4 * 90.0)
    b, f = one(kind, case["paths"], case.get("nS", 0), case.get("nT", 0),
               40 if kind == "multi" else case.get("steps", 1), case.get("payoffs", 1))
    return dict(bytes=b, flops=f)


# ---------------------------------------------------------------------------------------
# exact(): the same mathematics in 64-bit torch
# ---------------------------------------------------------------------------------------
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


M1, M2 = 4294967087, 4294944443


def _mulmod(a, b, m):
    """a b mod m for whole numbers below 2^32 (b a Python int)."""
    return (((a >> 16) * b % m) * 65536 + (a & 65535) * b) % m


def _matpow(a, n, m):
    r = [[int(i == j) for j in range(3)] for i in range(3)]
    mul = lambda p, q: [[sum(p[i][k] * q[k][j] for k in range(3)) % m for j in range(3)] for i in range(3)]  # noqa: E731
    while n:
        if n & 1:
            r = mul(r, a)
        a, n = mul(a, a), n >> 1
    return r


def _inv_normal(p, upper):
    """Beasley-Springer-Moro: p is the uniform's distance from the nearer end of [0, 1]."""
    x = p - 0.5
    r = x * x
    mid = x * (((-25.44106049637 * r + 41.39119773534) * r - 18.61500062529) * r + 2.50662823884) / (
        (((3.13082909833 * r - 21.06224101826) * r + 23.08336743743) * r - 8.47351093090) * r + 1.0)
    t = torch.log(-torch.log(p))
    q = torch.zeros_like(t)
    for c in (0.0000003960315187, 0.0000002888167364, 0.0000321767881768, 0.0003951896511919, 0.0038405729373609,
              0.0276438810333863, 0.1607979714918209, 0.9761690190917186, 0.3374754822726147):
        q = q * t + c
    g = torch.where(x.abs() < 0.42, mid, -q)
    return torch.where(upper, -g, g)


def _mrg(seed1, seed2, dim, first, units):
    """Gaussians of units [first, first + units), one tensor per dimension."""
    idx = torch.arange(first, first + units, device=_dev())
    out = []
    for seed, m, a in ((seed1, M1, [[0, 1403580, M1 - 810728], [1, 0, 0], [0, 1, 0]]),
                       (seed2, M2, [[527612, 0, M2 - 1370589], [1, 0, 0], [0, 1, 0]])):
        s = [torch.full_like(idx, seed) for _ in range(3)]
        p, bit = _matpow(a, dim, m), 0
        while (first + units - 1) >> bit:
            t = [sum(_mulmod(s[k], p[i][k], m) for k in range(3)) % m for i in range(3)]
            on = (idx >> bit) & 1 == 1
            s = [torch.where(on, t[i], s[i]) for i in range(3)]
            p, bit = _matpow(p, 2, m), bit + 1
        out.append(s)
    x, y = out
    for _ in range(dim):
        x = [(1403580 * x[1] - 810728 * x[2]) % M1, x[0], x[1]]
        y = [(527612 * y[0] - 1370589 * y[2]) % M2, y[0], y[1]]
        d = torch.where(x[0] > y[0], x[0] - y[0], x[0] - y[0] + M1)
        upper = 2 * d > M1 + 1
        yield _inv_normal(torch.where(upper, M1 + 1 - d, d).double() / (M1 + 1), upper)


def _directions(dim):
    """Sobol direction numbers [bit][dimension] from the published initial values."""
    if "jk" not in _shared:
        with open(os.path.join(ROOT, "compfinance_gb300", "data", "sobol_joe_kuo.inc")) as f:
            text = f.read()
        _shared["jk"] = [[int(t.rstrip("u")) for t in line.replace("{", " ").replace("}", " ").replace(",", " ").split()]
                         for line in text.splitlines() if line.strip().startswith("{")]
    out = torch.zeros((32, dim), dtype=torch.int64)
    for d in range(dim):
        s, a, *ini = _shared["jk"][d]
        m = ini[:s] if s else [1] * 32
        for k in range(len(m), 32):
            v = m[k - s] ^ (m[k - s] << s)
            for j in range(1, s):
                if (a >> (s - 1 - j)) & 1:
                    v ^= m[k - j] << j
            m.append(v)
        out[:, d] = torch.tensor([(m[k] << (31 - k)) & 0xFFFFFFFF for k in range(32)])
    return out.to(_dev())


def _sobol(dim, first, n):
    """Gaussians of points first + 1 .. first + n of the sequence, one tensor per dimension."""
    idx = torch.arange(first + 1, first + n + 1, device=_dev())
    gray, dirs = idx ^ (idx >> 1), _directions(dim)
    bits = [b for b in range(32) if (first + n) >> b]
    on = [(gray >> b) & 1 for b in bits]
    for d in range(dim):
        s = torch.zeros_like(idx)
        for b, o in zip(bits, on):
            s ^= o * dirs[b, d]
        p = 2.3283064365387e-10 * s.double()  # the reference's truncated 2^-32
        yield _inv_normal(torch.where(p > 0.5, 1.0 - p, p), p > 0.5)


def _chunks(case, d, dim, most):
    """Consecutive path ranges: (paths, Gaussians per dimension, one value per path)."""
    n = case["paths"]
    for first in range(0, n, most):
        m = min(most, n - first)
        if case["sobol"]:
            yield m, _sobol(dim, first, m)
        else:
            u = (m + 1) // 2
            yield m, (torch.stack([g, -g], 1).reshape(-1)[:m] for g in _mrg(d["seed1"], d["seed2"], dim, first // 2, u))


def _fill(dates, max_dt):
    """Simulation dates: today and the product's, gaps above max_dt cut into equal parts."""
    seq = dates if dates[0] == 0.0 else [0.0] + dates
    out = [seq[0]]
    for nxt in seq[1:]:
        cur = out[-1]
        if nxt - cur > max_dt:
            h = (nxt - cur) / (int((nxt - cur) / max_dt - 1e-8) + 1)
            t = cur + h
            while t < nxt - 0.00136986301369863:
                out.append(t)
                t += h
        out.append(nxt)
    return out


class _Dupire:
    """Log-Euler paths on the local-vol grid, and the adjoint of the grid's values."""

    def __init__(self, m, dates):
        dev = _dev()
        self.tl = _fill(dates, m["max_dt"])
        self.n, self.nS, self.nT = len(self.tl) - 1, len(m["spots"]), len(m["times"])
        self.spot = m["spot"]
        self.X = torch.tensor(np.log(m["spots"]), device=dev)
        self.inv = 1.0 / (self.X[1:] - self.X[:-1])
        v = torch.tensor(m["vols"], device=dev)
        self.Y, self.cols = [], []
        for i in range(self.n):
            t, sq = self.tl[i], math.sqrt(self.tl[i + 1] - self.tl[i])
            k = int(np.searchsorted(m["times"], t, side="right"))
            if k == 0 or k == self.nT:
                c = 0 if k == 0 else self.nT - 1
                self.cols.append(((c, sq),))
                self.Y.append(sq * v[:, c])
            else:
                w = (t - m["times"][k - 1]) / (m["times"][k] - m["times"][k - 1])
                self.cols.append(((k - 1, sq * (1 - w)), (k, sq * w)))
                self.Y.append(sq * (v[:, k - 1] + (v[:, k] - v[:, k - 1]) * w))

    def vol(self, i, x):
        k = torch.searchsorted(self.X, x, right=True)
        inside = (k > 0) & (k < self.nS)
        j = (k - 1).clamp(0, self.nS - 2)
        t = torch.where(inside, (x - self.X[j]) * self.inv[j], (k > 0).double())
        y1, y2 = self.Y[i][j], self.Y[i][j + 1]
        return j, t, torch.lerp(y1, y2, t), torch.where(inside, (y2 - y1) * self.inv[j], 0.0)

    def paths(self, m, gauss):
        """The state at every date and the Gaussian of every step."""
        xs, gs = [torch.full((m,), math.log(self.spot), dtype=torch.float64, device=_dev())], []
        for i, g in enumerate(gauss):
            x = xs[-1]
            v = self.vol(i, x)[2]
            gs.append(g)
            xs.append(x + v * (g - 0.5 * v))
        return xs, gs

    def sweep(self, xs, gs, ax, seed_at, bucket=None, buckets=1):
        """Adjoints back to today from the seeds: ax at the last date of xs, more from seed_at(i).
        Returns [bucket][1 + nS nT]: to the spot and to every local vol."""
        row = torch.zeros((buckets, 1 + self.nS * self.nT), dtype=torch.float64, device=_dev())
        grid = row[:, 1:].view(buckets, self.nS, self.nT)
        at = 0 if bucket is None else bucket * self.nS
        for i in range(len(xs) - 2, -1, -1):
            j, t, v, slope = self.vol(i, xs[i])
            q = gs[i] - v
            av = ax * q
            ax = ax + av * slope
            s = torch.bincount(at + j, av * (1 - t), buckets * self.nS)
            s += torch.bincount(at + j + 1, av * t, buckets * self.nS)
            for c, w in self.cols[i]:
                grid[:, :, c] += w * s.view(buckets, self.nS)
            ax = ax + seed_at(i)
        row[:, 0] = torch.bincount(bucket, ax, buckets) / self.spot if bucket is not None else ax.sum() / self.spot
        return row


def _dates(u):
    out, t = [0.0], u["freq"]
    while u["maturity"] - t > 0.000114469:
        out.append(t)
        t += u["freq"]
    return out + [u["maturity"]]


def _exact_uoc(case, d, want):
    mdl, u, n = _Dupire(d["model"], _dates(d["uoc"])), d["uoc"], case["paths"]
    sm = d["model"]["spot"] * u["smooth"]
    top, bot = u["barrier"] + sm, u["barrier"] - sm
    dates = set(_dates(u))
    mon = [i for i, t in enumerate(mdl.tl) if t in dates]
    total, squares, risks, pays = torch.zeros(2, device=_dev()).double(), torch.zeros(2, device=_dev()).double(), 0.0, []
    for m, gauss in _chunks(case, d, mdl.n, 1 << 18):
        xs, gs = mdl.paths(m, gauss)
        dead = torch.zeros(m, dtype=torch.bool, device=_dev())
        alive, before = torch.ones(m, dtype=torch.float64, device=_dev()), {}
        for i in mon:
            S = xs[i].exp()
            dead |= S > top
            band = ~dead & (S > bot)
            if bool(band.any()):
                before[i] = (alive, band, S)
                alive = torch.where(band, alive * (top - S) / (2 * sm), alive)
        S = xs[-1].exp()
        euro = (S - u["strike"]).clamp(min=0.0)
        p = torch.stack([torch.where(dead, 0.0, alive * euro), euro], 1)
        total, squares = total + p.sum(0), squares + (p * p).sum(0)
        if want == "paths":
            pays.append(p)
        if want == "risk":
            adj = [torch.where(dead, 0.0, euro)]  # adjoint of the survival factor

            def at(i):
                if i not in before:
                    return 0.0
                was, band, Si = before[i]
                back = torch.where(band, -adj[0] * was / (2 * sm) * Si, 0.0)
                adj[0] = torch.where(band, adj[0] * (top - Si) / (2 * sm), adj[0])
                return back

            seed = torch.where(dead | ~(S > u["strike"]), 0.0, alive * S)
            risks = risks + mdl.sweep(xs, gs, seed + at(mdl.n), at)[0]
    if want == "paths":
        return torch.cat(pays)
    mean = total / n
    if want == "value":
        return dict(values=mean, stderrs=((squares / n - mean * mean).clamp(min=0.0) / n).sqrt())
    return dict(values=mean, value=float(mean[0]), risks=risks / n)


def _exact_multi(case, d):
    mats, strikes = d["portfolio"]
    every = sorted(set(mats))
    mdl, n = _Dupire(d["model"], every), case["paths"]
    ks = [sorted(k for m, k in zip(mats, strikes) if m == t) for t in every]
    at = [mdl.tl.index(t) for t in every]
    values, risks = [0.0] * len(every), [0.0] * len(every)
    for m, gauss in _chunks(case, d, mdl.n, 1 << 18):
        xs, gs = mdl.paths(m, gauss)
        for e, (i, k) in enumerate(zip(at, ks)):
            S, k = xs[i].exp(), torch.tensor(k, dtype=torch.float64, device=_dev())
            b = torch.searchsorted(k, S)  # strikes below the spot
            values[e] = values[e] + torch.stack([(S - x).clamp(min=0.0).sum() for x in k])
            r = mdl.sweep(xs[:i + 1], gs[:i], torch.where(b > 0, S, 0.0), lambda i: 0.0, b, len(k) + 1)
            risks[e] = risks[e] + r[1:].flip(0).cumsum(0).flip(0)
    return dict(values=torch.cat(values) / n, risks=torch.cat(risks).T.contiguous() / n)


def _exact_bs(case, d, risk):
    b, K, T, n = d["bs"], d["strike"], d["maturity"], case["paths"]
    par = torch.tensor([b["spot"], b["vol"], b["rate"], b["div"]], dtype=torch.float64, device=_dev(),
                       requires_grad=True)
    total = squares = 0.0
    for m, gauss in _chunks(case, d, 1, 1 << 20):
        g = next(iter(gauss))
        spot, vol, rate, div = par
        S = spot * torch.exp((rate - div - 0.5 * vol * vol) * T + vol * math.sqrt(T) * g)
        p = (S - K).clamp(min=0.0) * torch.exp(-rate * T)
        total, squares = total + p.sum(), squares + (p.detach() ** 2).sum()
    mean = total / n
    if not risk:
        mean = mean.detach()
        return dict(values=mean[None], stderrs=((squares / n - mean * mean).clamp(min=0.0) / n).sqrt()[None])
    grad = torch.autograd.grad(mean, par)[0]
    mean = mean.detach()
    return dict(values=mean[None], value=float(mean), risks=grad)


def _exact_md(case, d):
    m, nA, n = d["md"], 4, case["paths"]
    f = lambda v: torch.tensor(v, dtype=torch.float64, device=_dev()).reshape(-1)  # noqa: E731
    low = [(i, j) for i in range(nA) for j in range(i)]
    par = torch.cat([f(m["disc"]), f(m["spots"]), f(m["spreads"]), f(m["divs"]), f(m["atms"]), f(m["skews"]),
                     f([m["correl"][i][j] for i, j in low]), f(m["lam"])]).requires_grad_()
    nD = len(m["div_dates"])
    cut = np.cumsum([1, nA, nA, nD * nA, nA, nA, len(low)])
    disc, spots, spreads, divs, atms, skews, rho, lam = (par[a:b] for a, b in zip([0, *cut], [*cut, len(par)]))
    divs = divs.view(nD, nA)
    if case["kind"] == "autocall":
        a = W.MD4_AUTOCALL
        dates = np.cumsum([a["maturity"] / a["periods"]] * a["periods"]).tolist()
    else:
        dates = [W.MD4_BASKET["maturity"]]
    beta = atms + 2 * skews
    kinds = ["log" if abs(k) < 1e-5 else "normal" if abs(b) < 1e-5 else "sur" if b > 0 else "sub"
             for k, b in zip(skews.tolist(), beta.tolist())]
    alpha = [0.0 if k == "log" else -2 * spots[i] * skews[i] / (1.0 if k == "normal" else beta[i].abs())
             for i, k in enumerate(kinds)]
    cor = torch.eye(nA, dtype=torch.float64, device=_dev())
    for (i, j), r in zip(low, rho):
        e = torch.zeros_like(cor)
        e[i, j] = e[j, i] = 1.0
        cor = cor + e * (lam * (1 - r) + r)
    L = torch.linalg.cholesky(cor)
    total = grad = 0.0
    for c, gauss in _chunks(case, d, nA * len(dates), 1 << 17):
        g = torch.stack(list(gauss)).view(len(dates), nA, c)
        s, alive, pay, t0 = [spots[i] for i in range(nA)], 1.0, 0.0, 0.0
        for e, t in enumerate(dates):
            dt, w, new = t - t0, L @ g[e], []
            for i, k in enumerate(kinds):
                ff = torch.exp((disc[0] - spreads[i]) * dt)
                for q, at in enumerate(m["div_dates"]):
                    if t0 <= at < t:
                        ff = ff * (1 - divs[q, i])
                fwd, b = s[i] * ff, -beta[i] if k == "sub" else beta[i]
                sd = (alpha[i] if k == "normal" else -b if k == "sub" else b) * math.sqrt(dt)
                grow = 0 if k == "normal" else torch.exp(-0.5 * b * b * dt + sd * w[i])
                new.append(fwd + sd * w[i] if k == "normal" else fwd * grow if k == "log" else
                           (fwd + alpha[i]) * grow - alpha[i] if k == "sur" else (fwd - alpha[i]) * grow + alpha[i])
            s, t0, num = new, t, torch.exp(disc[0] * t)
            if case["kind"] == "basket":
                b = sum(x * y for x, y in zip(W.MD4_BASKET["weights"], s))
                pay = torch.stack([(b - k).clamp(min=0.0) / num for k in W.MD4_BASKET["strikes"]])
                continue
            worst = torch.stack([x / r for x, r in zip(s, a["refs"])]).min(0).values
            pay = pay + alive * a["cpn"] * (a["maturity"] / a["periods"]) / num
            if e + 1 < len(dates):
                surv = alive * ((a["ko"] + a["smooth"] - worst) / 2 / a["smooth"]).clamp(0.0, 1.0)
                pay, alive = pay + (alive - surv) / num, surv
            else:
                pay = pay + alive / num - alive * (a["strike"] - worst).clamp(min=0.0) / a["strike"] / num
        p = pay.reshape(-1, c).sum(1)
        grad = grad + torch.autograd.grad(p[0], par, retain_graph=True)[0]
        total = total + p.detach()
    return dict(values=total / n, value=float(total[0] / n), risks=grad / n)


def _exact(case, d):
    kind = case["kind"]
    if kind in ("bs_value", "bs_risk"):
        return _exact_bs(case, d, kind == "bs_risk")
    if kind in ("uoc_value", "uoc_risk", "uoc_paths"):
        return _exact_uoc(case, d, kind[4:])
    if kind == "multi":
        return _exact_multi(case, d)
    return _exact_md(case, d)


def _numpy(v):
    return {k: _numpy(x) for k, x in v.items()} if isinstance(v, dict) else v.cpu().numpy() if torch.is_tensor(v) else v


def exact(case, seed):
    d, kind = _inputs(case, seed), case["kind"]
    if kind == "superbucket":
        return None  # see listed(): its vegas depend on the rounding of the calibration's prices
    if kind != "serve":
        return _numpy(_exact(case, d))
    values, stderrs, risks = [], [], []
    for r in d["requests"]:
        one = dict(r, kind={"value": "bs_value", "risk": "uoc_risk", "multi": "multi"}[r["kind"]])
        x = dict(seed1=d["seed1"], seed2=d["seed2"])
        if r["kind"] == "value":
            x.update(bs=d["bs"], strike=r["strike"], maturity=1.0)
        elif r["kind"] == "risk":
            x.update(model=d["models"][r["grid"]], uoc=_barrier(r["steps"], r["strike"], r["barrier"]))
        else:
            x.update(model=dict(d["models"][r["grid"]], max_dt=MONTH), portfolio=_portfolio(r["payoffs"]))
        got = _numpy(_exact(one, x))
        values.append(got["values"])
        if r["kind"] == "value":
            stderrs.append(got["stderrs"])
        else:
            risks.append(got["risks"].reshape(-1))
    return dict(values=np.concatenate(values), stderrs=np.concatenate(stderrs) if stderrs else np.zeros(0),
                risks=np.concatenate(risks) if risks else np.zeros(0))
