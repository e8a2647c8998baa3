"""The walk in direction order (32 neighbouring rays per warp in step) at the
sizes and inputs where it can go wrong, against the oracle's maps: items one
ray short of, equal to and one over a CTA's rays; clouds with no order, with
many equal rays, and with rays that the loop must drop, clip or end early;
sensors at the window's edge, outside it and past its wrap; every layout.
Counts are whole numbers, so the maps must be equal bit for bit."""
import numpy as np
import pytest

import cublox_b200 as C
import oracle as O

pytestmark = pytest.mark.gpu

LO = C.yaml_log_odds()
SHAPES = (0, 2, 3, 4)  # batch launch shapes that walk in direction order


def _rays(rng, n, sensor, reach):
    d = rng.normal(size=(n, 3))
    d[:, 2] *= 0.3
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return (sensor + d * rng.uniform(0.01, reach, (n, 1))).astype(np.float32)


def _clouds(rng, n, sensor):
    """A cloud of n rays with no order, its special rays first."""
    p = _rays(rng, n, sensor, 9.0)
    s = np.asarray(sensor, np.float32)
    special = [s, s + [1e-7, 0, 0], s + [3, 0, 0], s - [0, 4, 0], s + [0, 0, 2], s + [2, 2, 0], s - [2, 2, 2],
               [np.nan, 0, 0], [np.inf, 1, 1], s + [1e-3, 5, 1e-30], s + [1e30, 0, 0], s + [40, 0.05, 0.05]]
    p[: min(n, len(special))] = np.asarray(special, np.float32)[: min(n, len(special))]
    if n > 600:
        p[-200:] = p[-1]  # many equal rays
    if n > 2000:
        p[600:1800] = np.nan  # items without a point
    return p


def _check(grid, half, ctr, sensors, clouds, update):
    o = O.OracleGrid(half, 0.1, ctr, 1.0)
    o.set_log_odds(*LO)
    o.set_max_range(6.0)
    for s, p in zip(sensors, clouds):
        update(p, s)
        o.update(p, s)
        assert np.array_equal(grid.export().view(np.uint32), o.occ().view(np.uint32))
        assert grid.recenter(s) == o.recenter(s)["action"]
    assert grid.check() == 0


@pytest.mark.parametrize("n", [1, 31, 33, 255, 256, 257, 511, 513, 1023, 1025, 3000])
def test_items_around_a_ctas_rays(n):
    half, rng = (37, 25, 11), np.random.default_rng(n)
    sensors = np.float32([[0.03, -0.02, 0.41], [1.9, -1.4, 0.6], [-30.0, 2.0, 0.3]])
    clouds = [_clouds(rng, n, s) for s in sensors]
    for shape in SHAPES:
        b = C.Batch()
        b.set_option(C.BATCH_OPT_SHAPE, shape)
        g = b.add_grid(half, 0.1, False, 1.0)
        g.setLogOddsParams(*LO)
        g.setMaxRaycastRange(6.0)
        g.enable_stats(shape == 2)  # the walk that counts, and the one that does not
        _check(g, half, False, sensors, clouds, lambda p, s: b.update([g], [p], [s]))
        b.close()


@pytest.mark.parametrize("layout", C.LAYOUTS)
@pytest.mark.parametrize("half", [(0, 0, 0), (3, 40, 2), (64, 5, 30)])
def test_window_edges_and_layouts(half, layout):
    """The sensor beside, on and outside the window's sides, after the window
    has wrapped around its ring buffer, for maps thin on one axis or more."""
    rng = np.random.default_rng(sum(half) + layout)
    b = C.Batch()
    b.set_option(C.BATCH_OPT_SHAPE, 0)
    b.set_option(C.BATCH_OPT_LAYOUT, layout)
    g = b.add_grid(half, 0.1, True, 1.0)
    g.setLogOddsParams(*LO)
    g.setMaxRaycastRange(6.0)
    edge = np.float32(half) * np.float32(0.1)
    sensors = np.float32([[0, 0, 0], edge, -edge + 0.04, edge * [1.2, 0, 0] + 0.06, [0.7, 0.6, 0.1], [5.1, -3.3, 0.2],
                          [5.1, -3.3 + 0.9, 0.2]])
    _check(g, half, True, sensors, [_clouds(rng, 700, s) for s in sensors], lambda p, s: b.update([g], [p], [s]))
    b.close()


def test_map_too_wide_for_the_step_table():
    half, rng = (2100, 1, 1), np.random.default_rng(4)
    b = C.Batch()
    b.set_option(C.BATCH_OPT_SHAPE, 0)
    g = b.add_grid(half, 0.1, False, 1.0)
    g.setLogOddsParams(*LO)
    g.setMaxRaycastRange(6.0)
    s = np.float32([[0.0, 0.0, 0.0]])
    _check(g, half, False, s, [_clouds(rng, 2000, s[0])], lambda p, x: b.update([g], [p], [x]))
    b.close()


@pytest.mark.parametrize("n", [1, 63, 64, 65, 4096, 32767, 32769, 65537, 131073, 262144])
@pytest.mark.parametrize("source", ["host", "device", "device_soa"])
def test_single_grid_items(n, source):
    """One grid's update at the sizes where its items get wider."""
    import torch

    half, rng = (40, 33, 14), np.random.default_rng(n)
    g = C.OccupancyGrid(half, 0.1, False, 1.0)
    g.setLogOddsParams(*LO)
    g.setMaxRaycastRange(6.0)
    sensors = np.float32([[0.03, -0.02, 0.41], [1.9, -1.4, 0.6]])
    keep = []

    def update(p, s):
        if source != "host":
            t = torch.from_numpy(p).cuda()
            keep.append(t if source == "device" else t.T.contiguous())
            torch.cuda.synchronize()
            if source == "device":
                g.update_ptr(keep[-1].data_ptr(), n, s, C.LAYOUT_AOS)
            else:
                g.update_ptr(keep[-1].data_ptr(), n, s, C.LAYOUT_SOA)
        else:
            g.update(p, s)

    _check(g, half, False, sensors, [_clouds(rng, n, s) for s in sensors], update)
    g.close()
