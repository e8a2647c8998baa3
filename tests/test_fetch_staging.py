"""Large fetches into pageable memory, whose pinned staging buffers outlive the
grids: a grid's first fetch pins none but rarely, never more than three in all;
fetches of several grids at once each have their own, and one that can have none
still gets its samples."""
import threading

import numpy as np
import pytest

import cublox_b200 as C

pytestmark = pytest.mark.gpu

HALF = (60, 60, 20)


def _grid(seed):
    g = C.OccupancyGrid(HALF, 0.1, False, None)
    g.import_(np.random.default_rng(seed).choice(np.float32([-1, 0, 2]), int(np.prod(2 * np.array(HALF) + 1))))
    return g


def _centres(n):
    return (np.random.default_rng(n).uniform(-3, 3, (n, 3)) * [1, 1, 0.2]).astype(np.float32)


def _alone(g, c):
    """The same fetch in pieces that the runtime copies."""
    parts = [g.fetch_batch(c[i:i + 10], 1.0) for i in range(0, len(c), 10)]
    return tuple(np.concatenate([p[k] for p in parts]) for k in (1, 2))


def test_staging_outlives_the_grid():
    c = _centres(150)  # 8 MB
    pinned = []
    for seed in range(6):
        g = _grid(seed)
        want = _alone(g, c)
        before = C.runtime_counters()["pinned_allocs"]
        _, pos, st = g.fetch_batch(c, 1.0)
        pinned.append(C.runtime_counters()["pinned_allocs"] - before)
        assert pos.nbytes + st.nbytes > 4 << 20
        assert np.array_equal(pos, want[0]) and np.array_equal(st, want[1])
        g.close()
    assert max(pinned) <= 1 and sum(pinned) <= 2, pinned  # the first, and at most one of the later ones


def test_grids_that_fetch_at_once():
    c = _centres(300)
    grids = [_grid(seed) for seed in range(5)]
    want = [_alone(g, c) for g in grids]
    bad = []

    def run(k):
        for _ in range(4):
            _, pos, st = grids[k].fetch_batch(c, 1.0)
            if not (np.array_equal(pos, want[k][0]) and np.array_equal(st, want[k][1])):
                bad.append(k)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(5)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    # three buffers are kept; the other grids' went back
    n = C.runtime_counters()
    C.fail_allocations(0, 1 << 20)
    try:
        for k in range(5):
            _, pos, st = grids[k].fetch_batch(c, 1.0)
            assert np.array_equal(pos, want[k][0]) and np.array_equal(st, want[k][1])
    finally:
        C.fail_allocations(0, 0)
    assert C.runtime_counters()["pinned_allocs"] == n["pinned_allocs"]
    for g in grids:
        g.close()


def test_no_memory_for_staging():
    """In a process of its own, where no buffer waits yet."""
    import subprocess
    import sys

    code = ("import numpy as np, cublox_b200 as C\n"
            "from tests.test_fetch_staging import _grid, _centres, _alone\n"
            "g, c = _grid(1), _centres(150)\n"
            "want = _alone(g, c)\n"
            "g.fetch_counts(c, 1.0)\n"  # the block and the offsets
            "L = C.lib()\n"
            "import ctypes\n"
            "F, I = ctypes.POINTER(ctypes.c_float), ctypes.POINTER(ctypes.c_int64)\n"
            "off = np.zeros(151, np.int64)\n"
            "assert L.cublox_grid_fetch_begin(g._h, c.ctypes.data_as(F), 150, 1.0, -1, 0, off.ctypes.data_as(I)) == 0\n"
            "pos = np.zeros((off[150], 3), np.float32)\n"
            "C.fail_allocations(0, 1000)\n"
            "assert L.cublox_grid_fetch_read(g._h, pos.ctypes.data_as(F), None, int(off[150])) == 0\n"
            "assert np.array_equal(pos, want[0])\n"
            "print('staged by the runtime')\n")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "staged by the runtime" in r.stdout, r.stderr
