"""Worst-of autocall with assets of exactly equal performance: the first of them takes the adjoint, as
the reference's min_element, whatever the references' reciprocals round to."""
import numpy as np
import pytest

import oracle as O
from compfinance_gb300 import Engine
from gpu_util import num, rel_to_max

pytestmark = pytest.mark.gpu

# spots and vols; the references are the spots, so an asset without vol stays at a performance of 1
BOOKS = [
    ([100.0, 49.0], [0.0, 0.0]),
    ([49.0, 100.0, 98.0, 103.0], [0.0, 0.0, 0.0, 0.0]),
    ([107.0, 100.0, 49.0, 50.0], [0.0, 0.0, 0.0, 0.0]),
    ([100.0, 80.0, 49.0, 103.0], [0.2, 0.0, 0.0, 0.0]),   # one asset above or below the tied ones
    ([100.0, 49.0, 98.0, 50.0], [0.0, 0.25, 0.0, 0.0]),
    ([100.0, 49.0, 98.0, 103.0, 107.0, 50.0], [0.0] * 6),  # the wide form
]


@pytest.mark.parametrize("k", range(len(BOOKS)))
@pytest.mark.parametrize("sob", [0, 1])
def test_first_of_equal_performances(k, sob):
    spots, vols = BOOKS[k]
    n = len(spots)
    names = ["A%d" % i for i in range(n)]
    correl = np.eye(n) + 0.3 * (1 - np.eye(n))
    ms = dict(assets=names, spots=spots, atms=vols, skews=[0.0] * n, disc=0.0, spreads=[0.0] * n, div_dates=[], divs=[],
              correl=correl, **{"lambda": 0.0})
    # the put's strike above 1: the worst asset's adjoint is not zero at the last date
    ps = dict(kind="autocall", assets=names, refs=spots, maturity=2.0, periods=4, ko=1.05, strike=1.1, cpn=0.06, smooth=0.1)
    eng = Engine(0)
    try:
        eng.putDisplaced(names, spots, vols, ms["skews"], 0.0, ms["spreads"], [], [], correl, 0.0, "m")
        eng.putAutocall(names, spots, 2.0, 4, ps["ko"], ps["strike"], ps["cpn"], ps["smooth"], "p")
        r = eng.AADriskOne("m", "p", num(sob, 2000))
        v, _, risks = O.m_risk(O.MModel(ms), O.MProduct(ps), sob, 2000, [1.0])
        assert np.abs(risks).max() > 0
        # path sums of some hundred operations per path
        assert rel_to_max(r["payoffValues"], v) <= 1e-12
        assert rel_to_max(r["risks"], risks) <= 1e-12
    finally:
        eng.close()
