"""Results written to the host by a run's last block (small runs) against those copied after it (large
ones): books on either side of the line at 64 accumulators, from one block to many, repeated and
alternated on one engine so that a result left over from the run before would show."""
import numpy as np
import pytest

import oracle as O
from compfinance_gb300 import Engine
from gpu_util import num, rel_to_max

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = Engine(0)
    e.putBlackScholes(100.0, 0.2, 0, 0.02, 0.01, "m")
    yield e
    e.close()


# accumulators: two per payoff and two, and four more in a risk run
@pytest.mark.parametrize("npay", [1, 28, 29, 30, 31, 32])
@pytest.mark.parametrize("n", [1, 127, 129, 40001])
def test_small_and_large_books(eng, npay, n):
    """Tolerance: a value's or adjoint's rounding errors on one path are some tens of units of 2^-53 of
    quantities no larger than ten times the spot; averages keep them below 1e-12 of it."""
    mats = [0.5 + 0.5 * (k % 4) for k in range(npay)]
    strikes = [80.0 + 1.5 * k for k in range(npay)]
    w = np.linspace(1.0, 2.0, npay)
    eng.putEuropeans(mats, strikes, "p")
    m = O.Model(dict(kind="bs", spot=100.0, vol=0.2, qspot=0, rate=0.02, div=0.01))
    p = O.Product(dict(kind="europeans", mats=mats, strikes=strikes))
    for seed1 in (12345, 777):
        values, risks = O.risk_multi(m, p, 0, n, seed1=seed1)
        values, risks = np.asarray(values), np.asarray(risks)
        x = eng.value("m", "p", num(0, n, seed1=seed1))
        assert np.abs(np.asarray(x["values"]) - values).max() <= 1e-12 * 100.0
        r = eng.AADriskAggregate("m", "p", w, num(0, n, seed1=seed1))
        assert np.abs(np.asarray(r["payoffValues"]) - values).max() <= 1e-12 * 100.0
        assert rel_to_max(r["risks"], risks @ w) <= 1e-12
