"""FP64 Dupire risk where a level is today's spot: the ends of a barrier's smoothing band (a product's first date
is today), and the strikes of a portfolio on a model without vol.  The slope there is one side's or the
other's; the reference takes the one that its doubles compare to, and so does the engine."""
import numpy as np
import pytest

import oracle as O
from compfinance_gb300 import Engine
from compfinance_gb300 import workloads as W
from gpu_util import num, rel_to_max

pytestmark = pytest.mark.gpu

SPOTS = [100.0, 50.0, 8.852553055550057, 37.7, 80.0, 120.0, 99.99999999999999, 1.1]


@pytest.fixture(scope="module")
def eng():
    e = Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("spot", SPOTS)
@pytest.mark.parametrize("end", ["start of the band", "knock-out"])
@pytest.mark.parametrize("smooth", [0.05, 0.01, 0.1])
def test_band_ends_at_spot(eng, spot, end, smooth):
    """Tolerance: a double's rounding of log S per step (2^-51 of it), over sqrt(steps) steps, four
    deviations, times barrier / band width."""
    s, t, v = W.dupire_surface(20, 10)
    s = s * (spot / 100.0)
    barrier = spot * (1.0 + smooth) if end == "start of the band" else spot * (1.0 - smooth)
    eng.putDupire(spot, s, t, v, 0.25, "m")
    eng.putBarrier(spot, barrier, 1.0, 0.25, smooth, 0, "p")
    m = O.Model(dict(kind="dupire", spot=spot, spots=s, times=t, vols=v, maxdt=0.25))
    p = O.Product(dict(kind="uoc", strike=spot, barrier=barrier, maturity=1.0, freq=0.25, smooth=smooth, callput=0))
    w = np.array([1.0, 0.0])
    values, _, risks = O.risk(m, p, 0, 2000, w)
    r = eng.AADriskAggregate("m", "p", w, num(0, 2000))
    tol = 4 * np.sqrt(5.0) * 5.0 * 2.0 ** -51 * max(1.0, barrier / (2 * spot * smooth))
    assert np.abs(r["payoffValues"] - values).max() <= tol * spot
    assert rel_to_max(r["risks"], risks) <= 2 * tol


@pytest.mark.parametrize("spot", SPOTS)
def test_strikes_at_spot_without_vol(eng, spot):
    s, t, _ = W.dupire_surface(20, 10)
    s = s * (spot / 100.0)
    v = np.zeros((20, 10))
    strikes = [spot, np.nextafter(spot, 0.0), np.nextafter(spot, 2 * spot), spot * (1 + 1e-14), spot * (1 - 1e-14), 0.9 * spot]
    mats = [1.0] * 6
    eng.putDupire(spot, s, t, v, 0.25, "m")
    eng.putEuropeans(mats, strikes, "p")
    m = O.Model(dict(kind="dupire", spot=spot, spots=s, times=t, vols=v, maxdt=0.25))
    values, risks = O.risk_multi(m, O.Product(dict(kind="europeans", mats=mats, strikes=strikes)), 1, 300)
    r = eng.AADriskMulti("m", "p", num(1, 300))
    assert np.abs(r["values"] - values).max() <= 2.0 ** -50 * spot  # a rounding of the spot and of the difference
    # the spot risk of each strike: none or one
    assert np.abs(r["risks"][0] - risks[0]).max() <= 2.0 ** -50
