"""FP64 Dupire runs that cannot have the memory they want: the forms with large scratch (records of a
portfolio's paths, rings of a barrier's rounds) give way to those with little, with the same results, and
leave no error for the calls after them.  The device's memory pool is replaced by one of a few GB."""
import ctypes

import numpy as np
import pytest

from compfinance_gb300 import Engine
from compfinance_gb300 import workloads as W
from gpu_util import num, rel_to_max

pytestmark = pytest.mark.gpu


class _PoolProps(ctypes.Structure):  # CUmemPoolProps
    _fields_ = [("allocType", ctypes.c_int), ("handleTypes", ctypes.c_int), ("locationType", ctypes.c_int),
                ("locationId", ctypes.c_int), ("security", ctypes.c_void_p), ("maxSize", ctypes.c_size_t),
                ("reserved", ctypes.c_ubyte * 56)]


class _SmallPool:
    """Stream-ordered allocations come from a pool of `size` bytes."""

    def __init__(self, size):
        self.size, self.cu = size, ctypes.CDLL("libcuda.so.1")

    def __enter__(self):
        self.old, self.pool = ctypes.c_void_p(), ctypes.c_void_p()
        props = _PoolProps(allocType=1, locationType=1, locationId=0, maxSize=self.size)  # pinned, on the device
        assert self.cu.cuDeviceGetMemPool(ctypes.byref(self.old), 0) == 0
        assert self.cu.cuMemPoolCreate(ctypes.byref(self.pool), ctypes.byref(props)) == 0
        assert self.cu.cuDeviceSetMemPool(0, self.pool) == 0
        return self

    def __exit__(self, *a):
        assert self.cu.cuDeviceSetMemPool(0, self.old) == 0
        assert self.cu.cuMemPoolDestroy(self.pool) == 0  # its allocations stay valid until they are freed


def _put(eng):
    s, t, v = W.dupire_surface(20, 10)
    eng.putDupire(100.0, s, t, v, 1.0 / 12.0, "m")
    eng.putEuropeans([1.0, 1.0, 2.0, 3.0, 3.0], [90.0, 100.0, 110.0, 95.0, 120.0], "book")
    eng.putBarrier(105.0, 140.0, 3.0, 3.0 / 260, 0.01, 0, "uoc")
    eng.putBlackScholes(100.0, 0.2, 0, 0.02, 0.01, "bs")


def _runs(eng, what):
    w = np.array([1.0, -0.5, 2.0, 0.25, 1.0])
    big = num(0, 6000000)  # 3.9 GB of records; the barrier's ring takes 4.3 GB, its smaller form's scratch 1 GB
    if what == "multi":
        r = eng.AADriskMulti("m", "book", big)
        return r["values"], r["risks"]
    if what == "aggregate":
        r = eng.AADriskAggregate("m", "book", w, big)
        return r["payoffValues"], r["risks"]
    r = eng.AADriskOne("m", "uoc", num(0, 600000))
    return r["payoffValues"], r["risks"]


@pytest.mark.parametrize("what", ["multi", "aggregate", "barrier"])
def test_gives_way(what):
    """The two forms differ by a double's rounding of log S per step (2^-51 of it), over sqrt(steps) steps,
    four deviations; the barrier's band turns it into one of barrier / band width, twice."""
    eng = Engine(0)
    try:
        _put(eng)
        eng.AADriskMulti("m", "book", num(0, 1000))  # tables and small buffers
        eng.AADriskOne("m", "uoc", num(0, 1000))
        with _SmallPool(4 << 30):
            taken = _runs(eng, what)
            # the calls after it check the thread's last error
            eng.AADriskMulti("bs", "book", num(1, 1000))
            eng.gaussians(0, 12345, 1234, 4, 0, 10)
        free = _runs(eng, what)
        assert not np.array_equal(taken[1], free[1])  # not the same form
        steps = 260 if what == "barrier" else 36
        tol = 4 * np.sqrt(steps + 1) * np.log(100.0) * 2.0 ** -51
        band = 140.0 / (2 * 100.0 * 0.01) if what == "barrier" else 1.0
        assert rel_to_max(taken[0], free[0]) <= tol * band
        assert rel_to_max(taken[1], free[1]) <= 4 * tol * band
    finally:
        eng.close()


def test_aggregate_of_a_large_book():
    """3,500 strikes: more than the general portfolio kernel's sums hold on an SM, so the aggregate's smaller
    form is the single adjoint of the weighted book.  Tolerance as above."""
    eng = Engine(0)
    try:
        s, t, v = W.dupire_surface(20, 10)
        eng.putDupire(100.0, s, t, v, 1.0 / 12.0, "m")
        eng.putEuropeans([3.0] * 3500, list(np.linspace(60.0, 150.0, 3500)), "book")
        w = np.linspace(0.5, 1.5, 3500) / 3500
        eng.AADriskAggregate("m", "book", w, num(0, 1000))
        with _SmallPool(1 << 30):
            taken = eng.AADriskAggregate("m", "book", w, num(0, 2000000))  # 1.3 GB of records
        free = eng.AADriskAggregate("m", "book", w, num(0, 2000000))
        assert not np.array_equal(taken["risks"], free["risks"])
        tol = 4 * np.sqrt(37) * np.log(100.0) * 2.0 ** -51
        assert rel_to_max(taken["payoffValues"], free["payoffValues"]) <= tol
        assert rel_to_max(taken["risks"], free["risks"]) <= 4 * tol
    finally:
        eng.close()
