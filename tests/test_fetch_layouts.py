"""Sphere fetches in layouts whose bricks are not the tiles that a fetch reads:
long, flat and high ones.  Samples bit for bit the oracle's."""
import numpy as np
import pytest

import cublox_b200 as C
import oracle as O

pytestmark = pytest.mark.gpu

LO = C.yaml_log_odds()


@pytest.mark.parametrize("layout", [500, 410, 140, 50, 311, 122, 113, 23, 41, 203, 5, 14])
def test_layouts_of_any_bricks(layout):
    half, rng = (31, 31, 15), np.random.default_rng(layout)  # whole bricks of every kind, nearly
    g, o = C.OccupancyGrid(half, 0.1, False, 4.0), O.OracleGrid(half, 0.1, False, 4.0)
    g.set_option(C.OPT_LAYOUT, layout)
    g.setLogOddsParams(*LO)
    o.set_log_odds(*LO)
    s = np.float32([1.93, -0.77, 0.35])  # a window that has wrapped
    p = (s + rng.normal(size=(4000, 3)) * np.float32([2.0, 2.0, 0.9])).astype(np.float32)
    g.update(p, s)
    o.update(p, s)
    centres = (s + rng.uniform(-2.5, 2.5, (5, 3)) * [1, 1, 0.4]).astype(np.float32)
    centres[0] = s
    for r, flt, cap in ((0.35, -1, 0), (1.4, 2, 0), (1.4, 1, 40), (3.0, -1, 0), (3.0, 0, 0)):
        off, pos, st = g.fetch_batch(centres, r, None if flt < 0 else flt, cap)
        want = [o.fetch(c, r, flt, cap) for c in centres]
        assert np.array_equal(np.diff(off), [len(w[0]) for w in want])
        assert np.array_equal(pos.view(np.uint32), np.concatenate([w[0] for w in want]).view(np.uint32))
        assert np.array_equal(st, np.concatenate([w[1] for w in want]))
    g.close()
