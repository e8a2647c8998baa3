"""cublox_grid_fetch_read gives the samples of the grid's last fetch_begin, and
refuses to give any other fetch's, also one of as many samples."""
import ctypes

import numpy as np
import pytest

import cublox_b200 as C

pytestmark = pytest.mark.gpu

F, I64, U8 = (ctypes.POINTER(t) for t in (ctypes.c_float, ctypes.c_int64, ctypes.c_uint8))
R = 0.35


def _fp(a):
    return a.ctypes.data_as(F)


def _others(L, g, c, n):
    """Every other fetch, around `c`, of n samples."""
    pos, st, off, got = np.empty((n, 3), np.float32), np.empty(n, np.uint8), np.zeros(2, np.int64), ctypes.c_int64()
    i64, u8 = off.ctypes.data_as(I64), st.ctypes.data_as(U8)
    return {
        "fetch": lambda: L.cublox_grid_fetch(g._h, _fp(c), R, -1, 0, _fp(pos), u8, n, ctypes.byref(got)),
        "fetch_batch": lambda: L.cublox_grid_fetch_batch(g._h, _fp(c), 1, R, -1, 0, i64, _fp(pos), u8, n),
        "fetch_counts": lambda: L.cublox_grid_fetch_counts(g._h, _fp(c), 1, R, -1, 0, i64),
        "fetch_viz": lambda: g.fetch_viz(c, R) is None,
    }


@pytest.mark.parametrize("other", ["fetch", "fetch_batch", "fetch_counts", "fetch_viz"])
def test_read_refuses_another_fetchs_samples(other):
    L = C.lib()
    g = C.OccupancyGrid((20, 20, 10), 0.1, False, None)
    a, b = np.float32([0.05, 0.05, 0.05]), np.float32([0.55, 0.55, 0.05])
    off = np.zeros(2, np.int64)

    def begin(c):
        assert L.cublox_grid_fetch_begin(g._h, _fp(c), 1, R, -1, 0, off.ctypes.data_as(I64)) == C.OK
        return int(off[1])

    n = begin(a)
    assert n > 0 and len(g.fetchOccupancyAround(b, R)[0]) == n  # as many samples around b
    pos = np.zeros((n, 3), np.float32)
    read = lambda: L.cublox_grid_fetch_read(g._h, _fp(pos), None, n)  # noqa: E731
    call = _others(L, g, b, n)[other]
    assert call() == C.OK  # no begin before it that read could mean
    assert read() == C.ERR_INVALID and not pos.any()
    begin(a)
    assert call() == C.OK
    assert read() == C.ERR_INVALID and not pos.any()
    begin(a), begin(b)
    for _ in range(2):
        assert read() == C.OK
        assert np.allclose(pos.mean(0), b, atol=1e-5)
    g.close()
