"""A fetch with too little capacity is refused without making room on the device
for the samples that nobody gets."""
import ctypes

import numpy as np
import pytest

import cublox_b200 as C

pytestmark = pytest.mark.gpu

F, I64 = ctypes.POINTER(ctypes.c_float), ctypes.POINTER(ctypes.c_int64)


@pytest.mark.parametrize("call", ["fetch", "fetch_batch"])
def test_refused_without_room_for_the_samples(call):
    L, g = C.lib(), C.OccupancyGrid((60, 60, 20), 0.1, False, None)
    c = np.float32([[0.05, 0.05, 0.05], [0.3, 0.2, 0.1]])
    pos, off, got = np.zeros((4, 3), np.float32), np.zeros(3, np.int64), ctypes.c_int64(7)
    small = {"fetch": lambda k: L.cublox_grid_fetch(g._h, c.ctypes.data_as(F), 1.5, -1, 0, pos.ctypes.data_as(F), None,
                                                    k, ctypes.byref(got)),
             "fetch_batch": lambda k: L.cublox_grid_fetch_batch(g._h, c.ctypes.data_as(F), 2, 1.5, -1, 0,
                                                                off.ctypes.data_as(I64), pos.ctypes.data_as(F), None,
                                                                k)}[call]
    before = C.runtime_counters()["device_allocs"]
    for k in (0, 4):
        assert small(k) == C.ERR_INVALID
    assert C.runtime_counters()["device_allocs"] - before == 1  # the query block
    assert not pos.any() and got.value in (0, 7)
    want, p, _ = g.fetch_batch(c, 1.5)
    if call == "fetch_batch":
        assert np.array_equal(off, want)
    assert small(4) == C.ERR_INVALID  # and once there is room
    assert not pos.any()
    assert np.array_equal(g.fetch_batch(c, 1.5)[1], p)
    g.close()
