"""The FP64 Dupire value and risk runs in fixed point (dupire_fx64) against the CPU oracle: path
counts at the edges of warps, rounds and blocks, both generators, the products it takes, grids and
vols at the limits of its ranges (beyond them the generic kernel answers), smoothing bands with
and without the series, adjoints beyond the shared slab's range."""
import numpy as np
import pytest

import oracle as O
from compfinance_gb300 import Engine
from compfinance_gb300 import workloads as W
from gpu_util import num, rel_to_max

pytestmark = pytest.mark.gpu

_even = lambda n: (np.array([50.0 * 4.0 ** (i / max(1, n - 1)) for i in range(n)]), np.linspace(0.1, 3.0, max(2, n // 2)))  # noqa: E731


def _grid(name):
    rs = np.random.RandomState(3)
    if name == "uneven":
        s, t = np.cumsum(rs.uniform(0.05, 6.0, 40)) + 40.0, np.array([0.2, 0.21, 1.0, 2.9])
    elif name == "on_knot":
        s, t = np.array([50.0, 80.0, 100.0, 120.0, 170.0]), np.array([0.5, 1.0, 2.0])
    elif name == "one_knot":
        s, t = np.array([90.0]), np.array([0.5, 2.0])
    else:
        s, t = _even({"20": 20, "60": 60, "120": 120}[name.split("_")[0]])
    v = np.maximum(0.05, 0.15 + 0.1 * np.exp(-t)[None, :] * np.log(s / 100.0)[:, None] ** 2
                   + 0.005 * rs.standard_normal((len(s), len(t))))
    return s, t, v * {"high": 8.0, "beyond": 60.0}.get(name.split("_")[-1], 1.0)


@pytest.fixture(scope="module")
def eng():
    e = Engine(0)
    yield e
    e.close()


def _uoc(steps=36, barrier=140.0, smooth=0.01, callput=0, strike=105.0):
    return dict(kind="uoc", strike=strike, barrier=barrier, maturity=3.0, freq=3.0 / steps, smooth=smooth, callput=callput)


CASES = [
    # grid, spot, product, paths, sobol, weights
    ("60", 100.0, _uoc(), 1, 0, (1, 0)),
    ("60", 100.0, _uoc(), 2, 1, (1, 0)),
    ("60", 100.0, _uoc(), 255, 0, (1, 0)),
    ("60", 100.0, _uoc(), 256, 1, (1, 0)),
    ("60", 100.0, _uoc(), 257, 0, (0.5, 2.0)),
    ("60", 100.0, _uoc(), 4097, 1, (0, 1)),
    ("120", 100.0, _uoc(52), 3001, 0, (1, 0)),           # blocks of 256
    ("20", 100.0, _uoc(1), 777, 1, (1, 0)),              # one step
    ("20", 100.0, _uoc(2), 777, 0, (1, 0)),
    ("60", 100.0, _uoc(callput=1, strike=110.0), 2000, 0, (1, 0)),
    ("60", 100.0, _uoc(smooth=0.2), 2000, 1, (1, 0)),    # band wider than the series takes
    ("60", 139.9, _uoc(), 2000, 0, (1, 0)),              # today's date in the band
    ("60", 150.0, _uoc(), 500, 1, (1, 1)),               # knocked out today
    ("60", 100.0, _uoc(smooth=0.0005), 4000, 0, (1, 0)),  # adjoints beyond the slab's range
    ("uneven", 100.0, _uoc(), 2000, 0, (1, 0)),
    ("on_knot", 100.0, _uoc(), 2000, 0, (1, 0)),         # today's spot on a knot: the interval above it
    ("one_knot", 100.0, _uoc(), 2000, 1, (1, 0)),
    ("60", 1.5, _uoc(barrier=2.1, strike=1.5), 500, 0, (1, 0)),  # far below the grid
    ("20_high", 100.0, _uoc(12), 2000, 0, (1, 0)),
    ("20_beyond", 100.0, _uoc(12), 500, 0, (1, 0)),      # the generic kernel
    ("60", 100.0, dict(kind="european", strike=100.0, exercise=1.0, settlement=1.0), 1, 0, (1,)),
    ("60", 100.0, dict(kind="european", strike=100.0, exercise=2.0, settlement=2.5), 5001, 0, (1,)),
    ("120", 100.0, dict(kind="european", strike=90.0, exercise=3.0, settlement=3.0), 1025, 1, (2.5,)),
    ("uneven", 100.0, dict(kind="european", strike=100.0, exercise=0.05, settlement=0.05), 333, 1, (1,)),
]


@pytest.mark.parametrize("k", range(len(CASES)))
def test_value_and_risk_against_the_oracle(eng, k):
    """Tolerance: a double's rounding of log S per step (2^-51 of it), over sqrt(steps) steps, four
    deviations; a barrier's band turns a relative error of the spot into one of barrier / band
    width in the survival factor, and two such factors may multiply."""
    grid, spot, prod, n, sob, w = CASES[k]
    s, t, v = _grid(grid)
    eng.putDupire(spot, s, t, v, 0.25, "m")
    if prod["kind"] == "uoc":
        eng.putBarrier(prod["strike"], prod["barrier"], prod["maturity"], prod["freq"], prod["smooth"], prod["callput"], "p")
    else:
        eng.putEuropean(prod["strike"], prod["exercise"], prod["settlement"], "p")
    m, p = O.Model(dict(kind="dupire", spot=spot, spots=s, times=t, vols=v, maxdt=0.25)), O.Product(prod)
    _, _, steps = O.shapes(m, p)
    tol = 4 * np.sqrt(steps + 1) * max(1.0, abs(np.log(spot))) * 2.0 ** -51
    band = prod["barrier"] / (2 * spot * min(prod["smooth"], 1.0)) if prod["kind"] == "uoc" else 1.0
    values, agg, risks = O.risk(m, p, sob, n, np.array(w, dtype=float))
    r = eng.AADriskAggregate("m", "p", np.array(w, dtype=float), num(sob, n))
    assert rel_to_max(r["payoffValues"], values) <= tol * max(1.0, band)
    assert abs(r["riskPayoffValue"] - agg) <= tol * max(1.0, band) * max(abs(agg), 1e-3 * spot)
    if np.abs(risks).max() > 0:
        assert rel_to_max(r["risks"], risks) <= 2 * tol * max(1.0, band)
    else:
        assert not np.any(r["risks"])
    x = eng.value("m", "p", num(sob, n))
    assert np.array_equal(x["values"], r["payoffValues"])
    y = eng.simulatePaths("m", "p", num(sob, n))
    assert rel_to_max(y.mean(axis=0), values) <= tol * max(1.0, band) + 1e-14


def _strikes(n, lo=70.0, hi=150.0):
    return [lo + (hi - lo) * i / max(1, n - 1) for i in range(n)]


PORTFOLIOS = [
    # grid, spot, [(maturity, strikes)], paths, sobol
    ("60", 100.0, [(0.5, _strikes(20)), (1.0, _strikes(20)), (3.0, _strikes(20))], 1, 1),
    ("60", 100.0, [(0.5, _strikes(5)), (2.0, _strikes(3))], 31, 0),
    ("60", 100.0, [(0.5, _strikes(5)), (2.0, _strikes(3))], 257, 0),
    ("20", 100.0, [(0.25 * k, _strikes(4)) for k in range(1, 17)], 1025, 1),   # 16 maturities
    ("120", 100.0, [(1.5, _strikes(40)), (3.0, _strikes(1))], 3000, 0),        # slab of 86 KB
    ("on_knot", 100.0, [(1.0, [100.0, 100.0, 90.0, 1e-3, 1e4]), (2.0, [100.0])], 2000, 1),  # equal and extreme strikes
    ("uneven", 100.0, [(0.01, [99.0, 101.0]), (0.02, [100.0])], 511, 1),
    ("one_knot", 80.0, [(1.0, _strikes(6))], 600, 0),
    ("20_beyond", 100.0, [(1.0, _strikes(3))], 300, 0),                        # multi_kernel
]


@pytest.mark.parametrize("k", range(len(PORTFOLIOS)))
def test_portfolio_against_the_oracle(eng, k):
    """Tolerance: as above; a payoff's relative error is that of the spot times spot / payoff, a node
    weight's that of log S over the smallest gap between knots."""
    grid, spot, book, n, sob = PORTFOLIOS[k]
    s, t, v = _grid(grid)
    mats = [m for m, ks in book for _ in ks]
    strikes = [x for _, ks in book for x in ks]
    eng.putDupire(spot, s, t, v, 0.25, "m")
    eng.putEuropeans(mats, strikes, "p")
    m = O.Model(dict(kind="dupire", spot=spot, spots=s, times=t, vols=v, maxdt=0.25))
    p = O.Product(dict(kind="europeans", mats=mats, strikes=strikes))
    npay, _, steps = O.shapes(m, p)
    values, risks = O.risk_multi(m, p, sob, n)
    tol = 4 * np.sqrt(steps + 1) * max(1.0, abs(np.log(spot))) * 2.0 ** -51
    gap = np.diff(np.log(s)).min() if len(s) > 1 else 1.0
    r = eng.AADriskMulti("m", "p", num(sob, n))
    assert np.abs(r["values"] - values).max() <= tol * spot * 4
    assert rel_to_max(r["risks"], risks) <= 2 * tol * (1 + 1 / gap)
    # the weighted book through the same kernels
    w = np.random.RandomState(1).uniform(-1, 2, npay)
    a = eng.AADriskAggregate("m", "p", w, num(sob, n))
    assert rel_to_max(a["risks"], r["risks"] @ w) <= 1e-12
    assert abs(a["riskPayoffValue"] - r["values"] @ w) <= 1e-12 * np.abs(w) @ r["values"]
