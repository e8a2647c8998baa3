"""Fetches whose query block is bounded: cut into groups of centres, centres
without level masks, and centres in parts, on a server's block of a fixed size,
on a grid's, and on the small one that a grid falls back on.  Samples bit for
bit the oracle's; a server allocates nothing within its configured limits, and
its least budget is what it was before the block held columns."""
import numpy as np
import pytest

import cublox_b200 as C
import oracle as O

pytestmark = pytest.mark.gpu

LO = C.yaml_log_odds()
FLAT = (235, 235, 3)  # a map whose whole layer is more columns than a small block holds


def _scan(rng, half, n=6000):
    s = np.float32([0.03, 0.01, 0.02])
    p = (s + rng.normal(size=(n, 3)) * np.float32(half) * np.float32([0.05, 0.05, 0.08])).astype(np.float32)
    return p, s


def _oracle(half, p, s):
    o = O.OracleGrid(half, 0.1, False, None)
    o.set_log_odds(*LO)
    o.set_max_range(30.0)
    o.update(p, s)
    return o


def _grid(half, p, s):
    g = C.OccupancyGrid(half, 0.1, False, None)
    g.setLogOddsParams(*LO)
    g.setMaxRaycastRange(30.0)
    g.update(p, s)
    return g


def _same(o, centres, r, flt, cap, off, pos, st):
    want = [o.fetch(c, r, flt, cap) for c in centres]
    assert np.array_equal(off, np.cumsum([0] + [len(w[0]) for w in want]))
    assert np.array_equal(pos.view(np.uint32), np.concatenate([w[0] for w in want]).view(np.uint32))
    assert np.array_equal(st, np.concatenate([w[1] for w in want]))


# radius, state, cap, centres: groups with masks and without, one centre without
# masks (in the middle of its window, where its box is the whole map), in parts
SERVED = [(2.0, 2, 0, 64), (2.0, -1, 50, 64), (1.0, 1, 0, 64), (23.4, -1, 0, 1), (23.4, 2, 0, 1), (23.4, 1, 0, 3),
          (15.0, 1, 0, 2), (15.0, 0, 7, 5), (0.05, -1, 0, 3)]


def test_served_fetches_of_any_radius_allocate_nothing():
    rng = np.random.default_rng(5)
    p, s = _scan(rng, FLAT)
    o = _oracle(FLAT, p, s)
    srv = C.Server(hbm_budget_bytes=1 << 30, max_tick_points=1 << 16, max_fetch_centres=64, max_fetch_samples=1 << 21)
    mid = srv.add_map(FLAT, 0.1, False, None, max_range=30.0, log_odds=LO)
    assert srv.wait(srv.submit_scan(mid, p, s, False)) == C.REQ_DONE
    srv.drain()
    before = C.runtime_counters()
    for r, flt, cap, n in SERVED:
        centres = (s + rng.uniform(-3, 3, (n, 3)) * [1, 1, 0.05]).astype(np.float32)
        centres[0] = s
        rid = srv.submit_fetch(mid, centres, r, None if flt < 0 else flt, cap)
        assert srv.wait(rid) == C.REQ_DONE
        _same(o, centres, r, flt, cap, *srv.fetch_result(rid, n))
        srv.release(rid)
    assert C.runtime_counters() == before
    srv.close()


@pytest.mark.parametrize("samples", [1, 1 << 18])
def test_served_fetches_of_more_samples_than_configured(samples):
    """Outputs too small to lend room to the block, and outputs whose lower half
    a fetch's samples do not fit: they are found again beside the block."""
    rng = np.random.default_rng(7)
    p, s = _scan(rng, FLAT)
    o = _oracle(FLAT, p, s)
    for r, flt, cap, n in [(1.5, -1, 0, 64), (15.0, 1, 0, 2), (23.4, -1, 0, 1), (2.0, 2, 0, 64), (23.4, 1, 0, 3)]:
        srv = C.Server(hbm_budget_bytes=1 << 30, max_tick_points=1 << 16, max_fetch_centres=64,
                       max_fetch_samples=samples, pinned_pool_bytes=1 << 24)
        mid = srv.add_map(FLAT, 0.1, False, None, max_range=30.0, log_odds=LO)
        assert srv.wait(srv.submit_scan(mid, p, s, False)) == C.REQ_DONE
        centres = (s + rng.uniform(-3, 3, (n, 3)) * [1, 1, 0.05]).astype(np.float32)
        centres[0] = s
        for _ in range(2):  # with room to make, and with room made
            rid = srv.submit_fetch(mid, centres, r, None if flt < 0 else flt, cap)
            assert srv.wait(rid) == C.REQ_DONE
            _same(o, centres, r, flt, cap, *srv.fetch_result(rid, n))
        srv.close()


def test_a_grids_block_is_bounded_and_small_where_memory_is_short():
    import torch

    rng = np.random.default_rng(6)
    p, s = _scan(rng, FLAT)
    o, g = _oracle(FLAT, p, s), _grid(FLAT, p, s)
    near = (s + rng.uniform(-2, 2, (64, 3)) * [1, 1, 0.05]).astype(np.float32)
    wide = np.repeat(near[:2], 80, 0)  # 160 boxes of 440 x 440 columns
    for cap in (0, 3):
        _same(o, near, 2.0, 1, cap, *g.fetch_batch(near, 2.0, 1, cap))
    free = torch.cuda.mem_get_info()[0]
    off, pos, st = g.fetch_batch(wide, 23.0, 2, 3)
    counts = g.fetch_counts(wide, 23.0, 2, 3)
    assert free - torch.cuda.mem_get_info()[0] <= 68 << 20
    _same(o, near[:1], 23.0, 2, 3, off[:2], pos[:off[1]], st[:off[1]])
    _same(o, near[1:2], 23.0, 2, 3, off[80:82] - off[80], pos[off[80]:off[81]], st[off[80]:off[81]])
    assert np.array_equal(counts, np.diff(off))
    _same(o, near, 2.0, 1, 0, *g.fetch_batch(near, 2.0, 1, 0))
    g.close()
    g = _grid(FLAT, p, s)
    C.fail_allocations(1, 1)  # not the offsets in pinned memory, but the block
    try:
        off, pos, st = g.fetch_batch(wide[:3], 23.0, 1, 0)
    finally:
        C.fail_allocations(0, 0)
    _same(o, wide[:3], 23.0, 1, 0, off, pos, st)
    C.fail_allocations(0, 1 << 20)
    try:
        with pytest.raises(C.CubloxError) as e:
            g.fetch_batch(wide, 23.0, 1, 0)  # more than the small block: not to be had either
        assert e.value.code == C.ERR_NOMEM
    finally:
        C.fail_allocations(0, 0)
    _same(o, near, 2.0, -1, 0, *g.fetch_batch(near, 2.0))
    g.close()


@pytest.mark.parametrize("points,centres,samples", [(1 << 20, 1024, 1 << 22), (4096, 8, 1 << 10), (1 << 18, 100000, 1 << 20)])
def test_a_servers_least_budget(points, centres, samples):
    """12 B a point, 1 MiB of descriptors, 13 B a sample and 16 KiB, and for the
    query block of n centres 48 n + 160 (n + 5,120) bytes."""
    want = 12 * points + (1 << 20) + 48 * centres + 160 * (centres + 32 * 160) + 13 * samples + (16 << 10)
    assert C.Server.scratch_bytes(points, centres, samples) == want
