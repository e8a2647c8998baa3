"""The walk in direction order on coordinates and resolutions near the end of
the float range, against the oracle's maps bit for bit."""
import numpy as np
import pytest

import cublox_b200 as C
import oracle as O

pytestmark = pytest.mark.gpu

LO = C.yaml_log_odds()


def _same(half, res, max_range, s, p):
    """One grid's update and a batch's, in direction order."""
    s, p = np.float32(s), np.float32(p)
    o = O.OracleGrid(half, res, False, None)
    o.set_log_odds(*LO)
    o.set_max_range(max_range)
    g, b = C.OccupancyGrid(half, res, False, None), C.Batch()
    b.set_option(C.BATCH_OPT_SHAPE, 0)
    bg = b.add_grid(half, res, False, None)
    for x in (g, bg):
        x.setLogOddsParams(*LO)
        x.setMaxRaycastRange(max_range)
    o.update(p, s)
    g.update(p, s)
    b.update([bg], [p], [s])
    assert np.count_nonzero(o.occ())
    for x in (g, bg):
        assert np.array_equal(x.export().view(np.uint32), o.occ().view(np.uint32))
    g.close()
    b.close()


@pytest.mark.parametrize("n", [1, 64, 700])
def test_points_whose_coordinates_add_up_to_infinity(n):
    """An item all of whose points have x + y + z out of range, 5 m above a
    sensor as far out: rays like any other."""
    _same((4, 4, 4), 1e30, 100.0, [2e38, 2e38, 0.0], [[2e38, 2e38, 5.0]] * n)


@pytest.mark.parametrize("res,max_range", [(2.476250399962677e38, 3e38), (1e25, 3e38), (9e24, 3e38)])
@pytest.mark.parametrize("n", [1, 65])
def test_times_that_run_out_of_range(n, res, max_range):
    """A ray that steps past its endpoint on voxels as long as the float range:
    no axis has a finite time left, and the rule picks one that the ray does not
    move on.  From 1e25 m on, maps are walked step by step."""
    s = [-2.83568231e18, 1.00390983e9, 0.0]
    _same((3, 3, 3), res, max_range, s, [[0.0, -0.0, 0.0]] * n)


LOW, TOP = -2**31, 2**31 - 1


@pytest.mark.parametrize("ctr", [False, True])
@pytest.mark.parametrize("win,sensor", [
    ((0, 0, 0), (-3e8, 0, 0)), ((0, 0, 0), (0, -3e8, 0)), ((LOW, 0, 0), (-3e8, 0, 0)), ((LOW, 0, 0), (3e8, 0, 0)),
    ((LOW, LOW, LOW), (-2.1474836e8, -2.1474836e8, -2.1474836e8)), ((TOP, 5, 0), (-3e8, 0, 0)), ((TOP, 5, 0), (3e8, 0, 0)),
    ((TOP, 0, 0), (2.1474836e8, 0.05, 0.05)), ((LOW + 3, 0, TOP - 2), (-2.1474835e8, 0.05, 2.1474835e8))], ids=str)
def test_indices_at_the_ends_of_their_range(win, sensor, ctr):
    """Sensors and windows 2^31 voxels from the origin and from one another: an
    index saturates, and its distance from the window wraps around.  As the
    walk of one thread a ray has it, which follows each axis's slot.  No ray
    reaches the last window."""
    half, rng = (20, 15, 6), np.random.default_rng(1)
    s = np.float32(sensor)
    d = rng.normal(size=(200, 3)) * 200
    d[:50] *= [1, 1e-3, 1e-3]
    d[50:100] *= [1e-3, 1, 1e-3]
    p = (s + d).astype(np.float32)
    ref, g, b = C.OccupancyGrid(half, 0.1, ctr, None), C.OccupancyGrid(half, 0.1, ctr, None), C.Batch()
    ref.set_option(C.OPT_RAYCAST, 0)
    b.set_option(C.BATCH_OPT_SHAPE, 0)
    bg = b.add_grid(half, 0.1, ctr, None)
    for x in (ref, g, bg):
        x.setLogOddsParams(*LO)
        x.setMaxRaycastRange(1e9)
        x.set_origin_index(win)
    ref.update(p, s)
    g.update(p, s)
    b.update([bg], [p], [s])
    want = ref.export().view(np.uint32)
    assert np.count_nonzero(want) or win == (LOW + 3, 0, TOP - 2)
    for x in (g, bg):
        assert np.array_equal(x.export().view(np.uint32), want)
    if win == (0, 0, 0):  # no index wraps around on the way
        o = O.OracleGrid(half, 0.1, ctr, None)
        o.set_log_odds(*LO)
        o.set_max_range(1e9)
        o.set_origin_index(win)
        o.update(p, s)
        assert np.array_equal(want, o.occ().view(np.uint32))
    for x in (ref, g):
        x.close()
    b.close()
