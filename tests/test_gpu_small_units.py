"""Sums of many small terms of one sign: a run in units of 2^-15 of the currency (a deep in-the-money payoff
of 0.0024 on every path, thousands of paths per block) against the same run in the currency itself."""
import numpy as np
import pytest

from compfinance_gb300 import Engine
from gpu_util import num

pytestmark = pytest.mark.gpu

U = 2.0 ** -15
# Black-Scholes and the lognormal basket scale exactly (multiplications by a power of two), up to
# the rounding of every term to 2^-60, 2^-61 / U in the currency.  A Dupire path takes log S,
# whose rounding is 2^-51 of it at either scale, over sqrt(13) steps, four deviations.
EXACT = 2.0 ** -43
DUPIRE = 4 * np.sqrt(13.0) * 6.0 * 2.0 ** -51


@pytest.fixture(scope="module")
def eng():
    e = Engine(0)
    yield e
    e.close()


def _risk_scale(params):  # d value / d spot does not scale, every other derivative does
    return np.array([1.0 if p.startswith("spot") else U for p in params])


def _compare(small, big, scale, tol):
    assert np.abs(small["payoffValues"] / U - big["payoffValues"]).max() <= tol * 100.0
    a, b = small["risks"] / scale, np.asarray(big["risks"])
    assert np.abs(a - b).max() <= tol * max(1.0, np.abs(b).max())


@pytest.mark.parametrize("sob", [0, 1])
def test_black_scholes(eng, sob):
    r = []
    for u in (U, 1.0):
        eng.putBlackScholes(100.0 * u, 0.2, 0, 0.02, 0.01, "m")
        eng.putEuropean(20.0 * u, 1.0, 1.0, "p")
        r.append(eng.AADriskOne("m", "p", num(sob, 1 << 23)))
        v = eng.value("m", "p", num(sob, 1 << 23))["values"]
        assert np.array_equal(v, r[-1]["payoffValues"])
    _compare(r[0], r[1], _risk_scale(eng.parameterLabels("m")), EXACT)


def test_basket(eng):
    r = []
    for u in (U, 1.0):
        eng.putDisplaced(["A", "B"], [100.0 * u, 80.0 * u], [0.2, 0.25], [0.0, 0.0], 0.02, [0.0, 0.0], [], [],
                         [[1.0, 0.4], [0.4, 1.0]], 0.0, "m")
        eng.putBaskets(["A", "B"], [0.6, 0.5], 1.0, [20.0 * u], "p")
        r.append(eng.AADriskOne("m", "p", num(1, 1 << 23)))
    _compare(r[0], r[1], _risk_scale(eng.parameterLabels("m")), EXACT)


def _dupire(eng, u, knots):
    s, t = np.array(knots) * u, np.array([0.25, 0.5, 1.0, 2.0])
    eng.putDupire(100.0 * u, s, t, np.full((len(s), len(t)), 0.2), 1.0 / 12.0, "m")


WIDE = [60.0, 80.0, 95.0, 105.0, 130.0, 170.0]
CLOSE = [60.0, 80.0, 95.0, 95.0 * (1.0 + 2.0 ** -40), 105.0, 130.0, 170.0]  # too close for the fixed point


def test_dupire_european(eng):
    r = []
    for u in (U, 1.0):
        _dupire(eng, u, WIDE)
        eng.putEuropean(20.0 * u, 1.0, 1.0, "p")
        r.append(eng.AADriskOne("m", "p", num(0, 1 << 23)))
    _compare(r[0], r[1], _risk_scale(eng.parameterLabels("m")), DUPIRE)


@pytest.mark.parametrize("knots", [WIDE, CLOSE])
def test_portfolio(eng, knots):
    r = []
    for u in (U, 1.0):
        _dupire(eng, u, knots)
        eng.putEuropeans([0.5, 0.5, 1.0], [100.0 * u, 105.0 * u, 95.0 * u], "p")
        r.append(eng.AADriskMulti("m", "p", num(1, 1 << 20)))
    a, b = r[0]["risks"] / _risk_scale(eng.parameterLabels("m"))[:, None], r[1]["risks"]
    assert np.abs(r[0]["values"] / U - r[1]["values"]).max() <= DUPIRE * 100.0
    # the node adjoints of a flat surface sum terms of both signs as large as ten times the largest
    assert np.abs(a - b).max() <= 10 * DUPIRE * np.abs(b).max()


def test_spot_risk_of_many_paths(eng):
    """Every path adds about 1 to the spot risk of a deep in-the-money option, straight into one pair of
    accumulators in the general portfolio kernel.  The flat surface's knots do not matter to it."""
    r = []
    for knots in (WIDE, CLOSE):
        _dupire(eng, 1.0, knots)
        eng.putEuropeans([0.25], [20.0], "p")
        r.append(eng.AADriskMulti("m", "p", num(0, 1 << 25)))
    assert np.abs(r[0]["values"] - r[1]["values"]).max() <= DUPIRE * 100.0
    assert abs(r[0]["risks"][0, 0] - r[1]["risks"][0, 0]) <= DUPIRE
