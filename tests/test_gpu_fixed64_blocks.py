"""FP64 Dupire risk in blocks of 384 threads, which a grid of many nodes takes when the run has more threads
than blocks of 128 keep resident (a 120x60 grid: two of either per SM): against the CPU oracle, both
generators and products, path counts that end within a warp, a block and a round."""
import numpy as np
import pytest

import oracle as O
from compfinance_gb300 import Engine
from compfinance_gb300 import workloads as W
from gpu_util import num, rel_to_max

pytestmark = pytest.mark.gpu

CASES = [
    # product, steps, paths, sobol, weights
    ("uoc", 12, 100001, 0, (1.0, 0.5)),
    ("uoc", 12, 262143, 0, (1.0, 0.0)),
    ("uoc", 12, 80003, 1, (1.0, 0.5)),
    ("uoc", 3, 400000, 1, (1.0, 0.0)),
    ("european", 8, 120002, 0, (1.0,)),
    ("european", 8, 80001, 1, (2.0,)),
]


@pytest.mark.parametrize("k", range(len(CASES)))
def test_large_blocks(k):
    """Tolerance: a double's rounding of log S per step (2^-51 of it), over sqrt(steps) steps, four
    deviations; the barrier's band turns it into one of barrier / band width, twice.  The oracle's own
    plain sums of n terms per step round by 2^-53 each."""
    kind, steps, n, sob, w = CASES[k]
    s, t, v = W.dupire_surface(120, 60)
    eng = Engine(0)
    try:
        eng.putDupire(100.0, s, t, v, 0.25, "m")
        if kind == "uoc":
            prod = dict(kind="uoc", strike=105.0, barrier=140.0, maturity=steps * 0.25, freq=0.25, smooth=0.01, callput=0)
            eng.putBarrier(105.0, 140.0, steps * 0.25, 0.25, 0.01, 0, "p")
        else:
            prod = dict(kind="european", strike=95.0, exercise=2.0, settlement=2.0)
            eng.putEuropean(95.0, 2.0, 2.0, "p")
        m, p = O.Model(dict(kind="dupire", spot=100.0, spots=s, times=t, vols=v, maxdt=0.25)), O.Product(prod)
        assert O.shapes(m, p)[2] == steps
        values, agg, risks = O.risk(m, p, sob, n, np.array(w))
        r = eng.AADriskAggregate("m", "p", np.array(w), num(sob, n))
        tol = 4 * (np.sqrt(steps + 1) * np.log(100.0) * 2.0 ** -51 + np.sqrt(n * steps) * 2.0 ** -53)
        band = 140.0 / (2 * 100.0 * 0.01) if kind == "uoc" else 1.0
        assert rel_to_max(r["payoffValues"], values) <= tol * band
        assert abs(r["riskPayoffValue"] - agg) <= tol * band * abs(agg)
        assert rel_to_max(r["risks"], risks) <= 2 * tol * band
    finally:
        eng.close()
