"""Sphere fetches at the sizes where their columns, tiles and levels end:
boxes of one voxel, of one brick more or less, of more than 32 levels, boxes
that wrap around the ring buffer (so far that both ends share a tile), every
layout, filter and cap, one centre and many, and outputs that a first fetch
has to make room for.  Bit for bit, in order, against the oracle."""
import numpy as np
import pytest

import cublox_b200 as C
import oracle as O

pytestmark = pytest.mark.gpu

LO = C.yaml_log_odds()


def _pair(half, ctr, origin, layout, rng):
    g, o = C.OccupancyGrid(half, 0.1, ctr, 4.0), O.OracleGrid(half, 0.1, ctr, 4.0)
    g.setLogOddsParams(*LO)
    o.set_log_odds(*LO)
    for x in (g, o):
        (x.setMaxRaycastRange if x is g else x.set_max_range)(6.0)
    if layout is not None:
        g.set_option(C.OPT_LAYOUT, layout)
    s = (np.float32(origin) * np.float32(0.1) + np.float32(0.03)).astype(np.float32)
    p = (s + rng.normal(size=(3000, 3)) * np.float32([2.0, 2.0, 0.7])).astype(np.float32)
    g.update(p, s)
    o.update(p, s)
    return g, o, s


def _same(g, o, centres, r, flt, cap):
    off, pos, st = g.fetch_batch(centres, r, None if flt < 0 else flt, cap)
    counts = g.fetch_counts(centres, r, None if flt < 0 else flt, cap)
    for i, c in enumerate(centres):
        op, os_, _ = o.fetch(c, r, flt, cap)
        assert counts[i] == len(op)
        assert np.array_equal(pos[off[i]:off[i + 1]].view(np.uint32), op.view(np.uint32))
        assert np.array_equal(st[off[i]:off[i + 1]], os_)


@pytest.mark.parametrize("layout", C.LAYOUTS)
@pytest.mark.parametrize("half,origin", [((20, 17, 9), (3, -4, 2)), ((9, 30, 40), (1000, 77, -35)),
                                         ((40, 3, 20), (-39, 2, 19))])
def test_fetch_tiles(half, origin, layout):
    rng = np.random.default_rng(sum(half) + layout)
    g, o, s = _pair(half, layout % 3 == 0, origin, layout, rng)
    centres = (s + rng.uniform(-1.2, 1.2, (7, 3)) * np.float32(half) * np.float32(0.1)).astype(np.float32)
    centres[0] = s
    for r in (0.04, 0.1, 0.35, 0.8, 3.9, 50.0):
        _same(g, o, centres, r, -1, 0)
    for flt, cap in ((0, 0), (1, 33), (2, 0), (-1, 1), (-1, 100)):
        _same(g, o, centres, 1.1, flt, cap)
    g.close()


def test_fetch_makes_room_and_keeps_it():
    rng = np.random.default_rng(8)
    half = (30, 30, 10)
    g, o, s = _pair(half, False, (0, 0, 0), None, rng)
    many = (s + rng.uniform(-2.0, 2.0, (1300, 3))).astype(np.float32)
    for centres, r in ((many[:1], 0.2), (many, 0.45), (many[:3], 2.0), (many[:1], 0.2), (many[:0], 1.0)):
        _same(g, o, centres, r, -1, 0)
    L = C.lib()
    import ctypes
    off, pos = np.zeros(2, np.int64), np.zeros((1, 3), np.float32)
    rc = L.cublox_grid_fetch_batch(g._h, many[0].ctypes.data_as(ctypes.POINTER(ctypes.c_float)), 1, 1.0, -1, 0,
                                   off.ctypes.data_as(ctypes.POINTER(ctypes.c_int64)),
                                   pos.ctypes.data_as(ctypes.POINTER(ctypes.c_float)), None, 1)
    assert rc == C.ERR_INVALID and not pos.any()  # too little room: refused, nothing written
    _same(g, o, many[:2], 0.3, -1, 0)
    g.close()


@pytest.mark.parametrize("n", [1, 127, 128, 129, 65536, 65537])
def test_query_in_place_and_copied(n):
    """Point queries where a CTA ends, and on both sides of the number of
    points that are read in place."""
    rng = np.random.default_rng(n)
    g, o, s = _pair((30, 30, 10), False, (7, -3, 2), None, rng)
    p = (s + rng.uniform(-3.5, 3.5, (n, 3))).astype(np.float32)
    p[0] = [np.nan, 0, 0]
    with np.errstate(invalid="ignore"):  # the reference bins on the host: x86 conversion, NaN to INT_MIN
        q = p * np.float32(1.0 / np.float32(0.1))
        v = np.where(np.isfinite(q), np.floor(q), -2.0**31).astype(np.int64)
    half, win = np.array((30, 30, 10)), np.array(o.origin()[0])
    inside = (np.abs(v - win) <= half).all(1)
    slot = (v + half) % (2 * half + 1)
    l = o.occ().reshape(2 * half + 1)[tuple(slot.T)]
    want = np.where(inside, np.where(l >= np.float32(LO[5]), 2, np.where(l < np.float32(LO[4]), 1, 0)), 0)
    for _ in range(2):
        assert np.array_equal(g.query_states(p), want)
    g.close()


def test_fetch_in_two_calls():
    """begin / read: samples of several copies' sizes, and what read refuses."""
    import ctypes

    rng = np.random.default_rng(2)
    g, o, s = _pair((60, 60, 20), False, (0, 0, 0), None, rng)
    L = C.lib()
    i64, f = ctypes.POINTER(ctypes.c_int64), ctypes.POINTER(ctypes.c_float)
    c = np.ascontiguousarray(s + rng.uniform(-1, 1, (40, 3)), np.float32)
    off = np.zeros(41, np.int64)
    for n, r in ((1, 0.3), (40, 0.5), (40, 2.0)):  # one piece, one copy, several threads
        assert L.cublox_grid_fetch_begin(g._h, c.ctypes.data_as(f), n, r, -1, 0, off.ctypes.data_as(i64)) == C.OK
        pos = np.empty((off[n], 3), np.float32)
        assert L.cublox_grid_fetch_read(g._h, pos.ctypes.data_as(f), None, int(off[n]) + 1) == C.ERR_INVALID
        for _ in range(2):
            assert L.cublox_grid_fetch_read(g._h, pos.ctypes.data_as(f), None, int(off[n])) == C.OK
        want = np.concatenate([o.fetch(x, r, -1, 0)[0] for x in c[:n]])
        assert np.array_equal(pos.view(np.uint32), want.view(np.uint32))
        g.fetch_counts(c, r)
        assert L.cublox_grid_fetch_read(g._h, pos.ctypes.data_as(f), None, int(off[n])) == C.ERR_INVALID
    g.close()
