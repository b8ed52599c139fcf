"""Reverse sweeps into a node slab held by spot row or by time column (multi_risk32.cu, mc_dupire_risk32.cuh,
fx_device.cuh): FP32 risks against FP64 ones of the same paths, and those against the CPU oracle, on grids
either side of the rule (a number of times divisible by eight or not), odd and even numbers of spots, one
spot, one time."""
import numpy as np
import pytest

import oracle as O
from compfinance_gb300 import Engine
from gpu_util import num, rel_to_max

pytestmark = pytest.mark.gpu

N = 2049


@pytest.fixture(scope="module")
def eng():
    e = Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("nS,nT", [(1, 4), (2, 1), (7, 3), (12, 4), (13, 12), (24, 16), (33, 8), (31, 31), (30, 32), (64, 6)])
def test_slab_layouts(eng, nS, nT):
    """Tolerances: FP64 as rounding allows, 1e-10 of the largest risk (knots no closer than 0.02 in log
    spot).  FP32: a path's log spot is off by some 1e-6, its weights on two knots by that over 0.02, and
    about one path in 10^5 per strike falls on the other side of it (at most one of 2049 here, worth
    1/2049 of a path's share of the risk times a few): 5e-3."""
    rs = np.random.RandomState(nS * 100 + nT)
    s = 100.0 * np.exp(0.02 * (np.arange(nS) - nS // 2) * min(4.0, 40.0 / nS + 1.0))
    t = np.linspace(0.2, 2.0, nT) if nT > 1 else np.array([1.0])
    v = 0.2 + 0.05 * rs.uniform(-1, 1, (nS, nT))
    eng.putDupire(100.0, s, t, v, 0.25, "m")
    mats, strikes = [0.5, 0.5, 1.0, 2.0, 2.0, 2.0], [95.0, 105.0, 100.0, 85.0, 100.0, 112.0]
    eng.putEuropeans(mats, strikes, "p")
    eng.putBarrier(100.0, 140.0, 2.0, 0.25, 0.02, 0, "u")
    m = O.Model(dict(kind="dupire", spot=100.0, spots=s, times=t, vols=v, maxdt=0.25))
    p = O.Product(dict(kind="europeans", mats=mats, strikes=strikes))
    _, risks = O.risk_multi(m, p, 1, N)
    r64 = eng.AADriskMulti("m", "p", num(1, N))["risks"]
    r32 = eng.AADriskMulti("m", "p", num(1, N, precision="fp32"))["risks"]
    assert rel_to_max(r64, risks) <= 1e-10
    assert rel_to_max(r32, r64) <= 5e-3
    u64 = eng.AADriskOne("m", "u", num(1, N))["risks"]
    u32 = eng.AADriskOne("m", "u", num(1, N, precision="fp32"))["risks"]
    u = O.Product(dict(kind="uoc", strike=100.0, barrier=140.0, maturity=2.0, freq=0.25, smooth=0.02, callput=0))
    assert rel_to_max(u64, O.risk(m, u, 1, N, np.array([1.0, 0.0]))[2]) <= 1e-10
    assert rel_to_max(u32, u64) <= 5e-3
