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
