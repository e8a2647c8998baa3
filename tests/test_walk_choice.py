"""One grid's scans on both sides of the rule that chooses between the walk in
direction order and the split walk, from every source of points: long and
short rays, few and many, maps too wide for the former's step table, sensors
and ranges that are no numbers.  Maps bit for bit the oracle's."""
import numpy as np
import pytest

import cublox_b200 as C
import oracle as O

pytestmark = pytest.mark.gpu

LO = C.yaml_log_odds()
# half size, rays, range: split (a corridor; few rays in a wide map), direction
# order (more rays, a shorter range, a shaft), split (no step table for the map)
SCANS = [((1500, 5, 4), 3000, 300.0), ((700, 600, 1), 900, 300.0), ((700, 600, 1), 40000, 300.0),
         ((1500, 5, 4), 3000, 20.0), ((4, 5, 1500), 3000, 300.0), ((2100, 1, 1), 2000, 300.0)]


def _cloud(rng, half, n, s):
    d = rng.normal(size=(n, 3)) * (np.float64(half) + 1)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return (s + d * rng.uniform(0.05, 0.11 * max(half), (n, 1))).astype(np.float32)


@pytest.mark.parametrize("source", ["pageable", "pinned", "device", "pageable soa", "device soa"])
@pytest.mark.parametrize("half,n,max_range", SCANS, ids=str)
def test_sources(half, n, max_range, source):
    import torch

    rng = np.random.default_rng(n)
    g, o = C.OccupancyGrid(half, 0.1, False, 1.0), O.OracleGrid(half, 0.1, False, 1.0)
    g.setLogOddsParams(*LO)
    g.setMaxRaycastRange(max_range)
    o.set_log_odds(*LO)
    o.set_max_range(max_range)
    for s in np.float32([[0.03, -0.02, 0.01], [1.3, 0.1, 0.05]]):
        p = _cloud(rng, half, n, s)
        t = torch.from_numpy(p.T.copy() if "soa" in source else p)
        t = t.cuda() if "device" in source else (t.pin_memory() if source == "pinned" else t)
        torch.cuda.synchronize()
        g.update_ptr(t.data_ptr(), n, s, C.LAYOUT_SOA if "soa" in source else C.LAYOUT_AOS)
        o.update(p, s)
        assert np.array_equal(g.export().view(np.uint32), o.occ().view(np.uint32))
        assert g.recenter(s) == o.recenter(s)["action"]
    assert g.check() == 0
    g.close()


@pytest.mark.parametrize("layout", C.LAYOUTS)
def test_split_walk_in_every_layout(layout):
    half, rng = (30, 24, 9), np.random.default_rng(layout)
    g, o = C.OccupancyGrid(half, 0.1, True, None), O.OracleGrid(half, 0.1, True, None)
    g.set_option(C.OPT_LAYOUT, layout)
    g.set_option(C.OPT_SEGMENT, 32)  # not the default: the split walk
    g.setLogOddsParams(*LO)
    o.set_log_odds(*LO)
    for s in np.float32([[0.0, 0.0, 0.0], [0.4, 0.3, 0.1]]):
        p = _cloud(rng, half, 3000, s)
        g.update(p, s)
        o.update(p, s)
        assert np.array_equal(g.export().view(np.uint32), o.occ().view(np.uint32))
    g.close()


@pytest.mark.parametrize("s", [(np.nan, 0, 0), (np.inf, 0, 0), (3e38, -3e38, 0), (0.05, 0.05, 0.05)], ids=str)
@pytest.mark.parametrize("max_range", [np.inf, np.nan, 0.0, -1.0, 1e-40, 3e38])
def test_sensors_and_ranges_at_the_ends(s, max_range):
    half, rng = (400, 400, 1), np.random.default_rng(3)
    g, o = C.OccupancyGrid(half, 0.1, False, None), O.OracleGrid(half, 0.1, False, None)
    for x, lo, mr in ((g, g.setLogOddsParams, g.setMaxRaycastRange), (o, o.set_log_odds, o.set_max_range)):
        lo(*LO)
        mr(max_range)
    p = _cloud(rng, (20, 20, 1), 300, np.zeros(3))
    g.update(p, np.float32(s))
    o.update(p, np.float32(s))
    assert np.array_equal(g.export().view(np.uint32), o.occ().view(np.uint32))
    g.close()


@pytest.mark.parametrize("away", [30.0, 2e4, 1e5])
def test_sensor_far_outside_the_window(away):
    """Rays that reach the window after 100 steps, or after hundreds of thousands."""
    half, rng = (30, 25, 8), np.random.default_rng(int(away))
    g, o = C.OccupancyGrid(half, 0.1, False, None), O.OracleGrid(half, 0.1, False, None)
    s = np.float32([away, 0.03, 0.05])
    p = (rng.normal(size=(200, 3)) * [1.5, 1.0, 0.4]).astype(np.float32)
    for x, lo, mr in ((g, g.setLogOddsParams, g.setMaxRaycastRange), (o, o.set_log_odds, o.set_max_range)):
        lo(*LO)
        mr(3e38)
        x.set_origin_index((0, 0, 0))
    g.update(p, s)
    o.update(p, s)
    assert np.count_nonzero(o.occ()) > 200
    assert np.array_equal(g.export().view(np.uint32), o.occ().view(np.uint32))
    assert g.check() == 0
    g.close()
