"""Shards of an FP64 run whose adjoints straddle the range of the shared node slab (a large notional): the
whole run takes blocks of 384 threads, its shards blocks of 128, and the sums agree bit for bit."""
import numpy as np
import pytest

from compfinance_gb300 import Engine, NumericalParam
from compfinance_gb300 import workloads as W
from compfinance_gb300.api import results_from_raw
from compfinance_gb300.shard import shard_range

pytestmark = pytest.mark.gpu


def _totals(acc):
    """The exact sums, units of 2^-60 (how they split into two words depends on the blocks), but the last, the
    aggregate's square: beyond 2^42 it has none."""
    return [(int(hi) << 40) + int(lo) for hi, lo in np.asarray(acc).reshape(-1, 2)[:-1]]


@pytest.mark.parametrize("prod", ["uoc", "european"])
@pytest.mark.parametrize("notional", [2.0e4, 4.0e5, 3.0e6])
def test_shards_of_a_large_notional(prod, notional):
    # 24 time columns for 520 steps: some 44 steps share a column, so the slab's range depends on the block
    s, t, v = W.dupire_surface(300, 24)
    eng = Engine(0)
    try:
        eng.putDupire(100.0, s, t, v, 3.0 / 520, "m")
        if prod == "uoc":
            eng.putBarrier(105.0, 150.0, 3.0, 3.0 / 520, 0.01, 0, "p")
        else:
            eng.putEuropean(100.0, 3.0, 3.0, "p")
        npay, npar, _ = eng.shapes("m", "p")
        w = np.full(npay, notional)
        n = 100000
        eng.enqueue("m", "p", NumericalParam(numPath=n, precision="fp64"), risk=True, weights=w)
        full, values = _totals(eng.fetch_raw()), eng.fetch(npay, npar)
        total = None
        for k in range(4):
            first, count = shard_range(n, k, 4)
            eng.enqueue_shard("m", "p", NumericalParam(numPath=count, precision="fp64"), first, risk=True, weights=w)
            acc = eng.fetch_raw()
            total = acc if total is None else total + acc
        assert _totals(total) == full and any(full)
        got = results_from_raw(total, npar, npay, n)  # sums beyond 2^33 among them: more than a double's bits
        assert np.array_equal(got[0], values[0]) and got[2] == values[2] and np.array_equal(got[3], values[3])
    finally:
        eng.close()
