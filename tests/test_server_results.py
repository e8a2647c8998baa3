"""Results of fetches that are not released, and scans: scans still find room in
the server's pinned arena (one that does not is kept in pageable memory until
its request is released, which shows in the process's resident memory), and
room that results held serves results of other sizes."""
import gc
import os

import numpy as np
import pytest

import cublox_b200 as C

pytestmark = pytest.mark.gpu

HALF = (40, 40, 12)


def _resident():
    with open("/proc/self/statm") as f:
        return int(f.read().split()[1]) * os.sysconf("SC_PAGE_SIZE")


def _server():
    s = C.Server(hbm_budget_bytes=2 << 30, max_tick_points=1 << 19, pinned_pool_bytes=16 << 20, max_fetch_centres=256,
                 max_fetch_samples=1 << 21)
    return s, s.add_map(HALF, 0.1, False, None, max_range=10.0, log_odds=C.yaml_log_odds())


@pytest.mark.parametrize("centres,fetches", [(200, 12), (1, 300)], ids=["large", "small"])
def test_scans_find_pinned_room_beside_unreleased_results(centres, fetches):
    rng = np.random.default_rng(1)
    s, mid = _server()
    at = rng.uniform(-1, 1, (centres, 3)).astype(np.float32) * np.float32([1, 1, 0.3])
    origin = np.float32([0.03, 0.02, 0.01])
    clouds = [(origin + rng.normal(size=(300000, 3))).astype(np.float32) for _ in range(2)]
    first = s.submit_scan(mid, clouds[0], origin, False)  # the map, the walk's shape, first-use memory
    for _ in range(14):
        s.wait(s.submit_scan(mid, clouds[0][:1000], origin, False))
    s.wait(first)
    s.release(first)
    ids = [s.submit_fetch(mid, at, 0.6) for _ in range(fetches)]
    for i in ids:
        assert s.wait(i) == C.REQ_DONE
    want = s.fetch_result(ids[0], centres)
    s.drain()
    gc.collect()
    before = _resident()
    for k in range(12):  # 12 x 3.6 MB, none released
        assert s.wait(s.submit_scan(mid, clouds[k % 2], origin, False)) == C.REQ_DONE
    grown = _resident() - before
    assert grown < 12 << 20, grown
    got = s.fetch_result(ids[-1], centres)
    for a, b in zip(want, got):
        assert np.array_equal(a, b)
    s.close()


def test_results_of_many_sizes_in_turn():
    """Held and released in every order: each reads what it fetched."""
    rng = np.random.default_rng(2)
    s, mid = _server()
    s.wait(s.submit_scan(mid, rng.normal(size=(5000, 3)).astype(np.float32), np.float32([0, 0, 0]), False))
    g = C.OccupancyGrid(HALF, 0.1, False, None)
    occ, _ = s.export(mid, int(np.prod(2 * np.array(HALF) + 1)))
    g.setLogOddsParams(*C.yaml_log_odds())
    g.import_(occ)
    held = []
    for k in range(60):
        n, r = int(rng.integers(1, 250)), float(rng.choice([0.15, 0.4, 0.7]))
        at = (rng.uniform(-2, 2, (n, 3)) * [1, 1, 0.2]).astype(np.float32)
        i = s.submit_fetch(mid, at, r)
        assert s.wait(i) == C.REQ_DONE
        held.append((i, at, r))
        while len(held) > 5:
            i, at, r = held.pop(int(rng.integers(len(held))))
            for a, b in zip(s.fetch_result(i, len(at)), g.fetch_batch(at, r)):
                assert np.array_equal(a, b)
            s.release(i)
    s.close()
    g.close()
