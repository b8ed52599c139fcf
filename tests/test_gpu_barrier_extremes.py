"""FP64 barriers at levels that are no ordinary number: what the double arithmetic of the comparisons says."""
import numpy as np
import pytest

from compfinance_gb300 import Engine
from compfinance_gb300 import workloads as W
from gpu_util import num

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def eng():
    e = Engine(0)
    s, t, v = W.dupire_surface(20, 10)
    e.putDupire(100.0, s, t, v, 0.25, "m")
    yield e
    e.close()


# barrier, smoothing, whether it ever knocks out
LEVELS = [(np.nan, 0.01, False), (150.0, np.nan, False), (np.inf, 0.01, False), (1e300, 0.01, False),
          (0.0, 0.01, True), (-50.0, 0.01, True), (1e-300, 0.01, True)]


@pytest.mark.parametrize("k", range(len(LEVELS)))
@pytest.mark.parametrize("sob", [0, 1])
def test_levels(eng, k, sob):
    barrier, smooth, out = LEVELS[k]
    eng.putBarrier(105.0, barrier, 1.0, 1.0 / 12.0, smooth, 0, "p")
    for v in (eng.value("m", "p", num(sob, 3000))["values"],
              eng.AADriskOne("m", "p", num(sob, 3000))["payoffValues"]):
        assert v[1] > 1.0  # the European
        assert v[0] == (0.0 if out else v[1])
