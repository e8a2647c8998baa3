"""Batches some of whose maps are too wide for the walk in direction order."""
import numpy as np
import pytest

import cublox_b200 as C
import oracle as O

pytestmark = pytest.mark.gpu

LO = C.yaml_log_odds()


def test_updates_with_and_without_a_wide_map_in_turn():
    """They replay a graph each: none is built again, and the maps are the
    oracle's."""
    rng = np.random.default_rng(1)
    halves = [(2100, 1, 1), (30, 20, 8), (25, 33, 5)]
    b = C.Batch()
    b.set_option(C.BATCH_OPT_GRAPHS, 1)
    b.set_option(C.BATCH_OPT_AUTOTUNE, 0)
    pairs = []
    for h in halves:
        g, o = b.add_grid(h, 0.1, False, None), O.OracleGrid(h, 0.1, False, None)
        g.setLogOddsParams(*LO)
        g.setMaxRaycastRange(6.0)
        o.set_log_odds(*LO)
        o.set_max_range(6.0)
        pairs.append((g, o))
    s = np.float32([0.01, 0.02, 0.03])

    def update(which):
        clouds = [(s + rng.normal(size=(700, 3)) * np.float32([2, 2, 0.5])).astype(np.float32) for _ in which]
        b.update([pairs[k][0] for k in which], clouds, np.stack([s] * len(which)))
        for k, c in zip(which, clouds):
            pairs[k][1].update(c, s)

    update([0, 1, 2])
    update([1, 2])
    b.synchronize()
    before = C.runtime_counters()["graph_builds"]
    for _ in range(3):
        update([1, 2])
        update([0, 1])
    assert C.runtime_counters()["graph_builds"] == before
    for g, o in pairs:
        assert np.array_equal(g.export().view(np.uint32), o.occ().view(np.uint32))
        assert g.check() == 0
    b.close()
