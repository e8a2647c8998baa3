"""Sphere fetches in every contraction mode of their distance test, on the
probe's queries, which tell the modes apart."""
import numpy as np
import pytest

import cublox_b200 as C
from tests import fp_probe as P

pytestmark = pytest.mark.gpu


def test_every_contraction_mode():
    pr = P.build_fetch_probe()
    g = C.OccupancyGrid(pr["half"], 0.1, False, None)
    g.set_origin_index((0, 0, 0))
    g.setLogOddsParams(*pr["lo"])
    g.import_(pr["occ"])
    seen = set()
    for mode, og in pr["grids"].items():
        g.set_fp_mode(mode)
        found = []
        for c, r in pr["queries"]:
            for flt in (None, 2):
                pos, st = g.fetchOccupancyAround(c, r, flt)
                want = og.fetch(c, r, -1 if flt is None else flt, 0)
                assert np.array_equal(pos.view(np.uint32), want[0].view(np.uint32))
                assert np.array_equal(st, want[1])
                found.append(len(st))
        seen.add(tuple(found))
    assert len(pr["grids"]) > 2 and len(seen) > 1  # the modes do differ here
    g.close()
