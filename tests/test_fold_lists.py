"""The fold of flagged lines at the sizes where its items end: maps of one
line, one line more or less than an item, and many items; scans whose lines
all hold a hit, or none.  Bit for bit against the oracle."""
import numpy as np
import pytest

import cublox_b200 as C
import oracle as O

pytestmark = pytest.mark.gpu

LO = C.yaml_log_odds()
# 8 x 4 x 1 bricks: lines = ceil(nx / 8) * ceil(ny / 4) * nz
HALVES = [(3, 1, 0), (3, 1, 7), (63, 31, 3), (63, 31, 4), (70, 60, 20)]


def _scan(rng, kind, half):
    span = (np.float32(half) + 0.4) * np.float32(0.1)
    if kind == "all hits":  # an endpoint in every voxel of the map's middle
        n = [2 * min(h, 20) + 1 for h in half]
        g = np.stack(np.meshgrid(*[np.arange(k) - k // 2 for k in n], indexing="ij"), -1).reshape(-1, 3)
        return (g * 0.1 + 0.01).astype(np.float32)
    d = rng.normal(size=(3000, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    if kind == "no hits":  # every ray clipped at max range
        return (d * 50.0).astype(np.float32)
    return (d * span * rng.uniform(0.1, 1.0, (3000, 1))).astype(np.float32)


@pytest.mark.parametrize("kind", ["all hits", "no hits", "mixed"])
@pytest.mark.parametrize("half", HALVES)
def test_items_and_hit_lines(half, kind):
    rng = np.random.default_rng(sum(half))
    s = np.float32([0.013, 0.021, 0.017])
    p = _scan(rng, kind, half)
    o = O.OracleGrid(half, 0.1, True, None)
    g = C.OccupancyGrid(half, 0.1, True, None)
    b = C.Batch()
    b.set_option(C.BATCH_OPT_SHAPE, 0)
    bg = b.add_grid(half, 0.1, True, None)
    o.set_log_odds(*LO)
    o.set_max_range(4.0)
    for x in (g, bg):
        x.setLogOddsParams(*LO)
        x.setMaxRaycastRange(4.0)
    for fold in (2, 3, 2):  # lists, flags per warp (it must leave no flag behind), lists
        o.update(p, s)
        g.set_option(C.OPT_FOLD, fold)
        b.set_option(C.BATCH_OPT_FOLD, 0 if fold == 2 else 2)
        g.update(p, s)
        b.update([bg], [p], [s])
        for x in (g, bg):
            assert np.array_equal(x.export().view(np.uint32), o.occ().view(np.uint32))
    g.close()
    b.close()
