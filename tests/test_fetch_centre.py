"""fetchOccupancyAround takes one centre, as the grid's other calls take a
position: up to three numbers in any sequence, those missing zero."""
import numpy as np
import pytest

import cublox_b200 as C


class _Calls(C.OccupancyGrid):
    """A grid without a device: records the centres of its fetch."""

    def __init__(self):
        self._h, self.centres = None, None

    def _fetch(self, centers, *args):
        self.centres = np.asarray(centers, np.float32).reshape(-1, 3)
        return None, None, None

    def close(self):
        pass


@pytest.mark.parametrize("centre,want", [((1, 2, 3), (1, 2, 3)), ([0.5, -2], (0.5, -2, 0)), ((), (0, 0, 0)),
                                         (np.float64([1e-3, 7, 9]), (1e-3, 7, 9)), (iter([4, 5, 6]), (4, 5, 6))])
def test_centres_taken(centre, want):
    g = _Calls()
    g.fetchOccupancyAround(centre, 1.0)
    assert np.array_equal(g.centres, np.float32([want]))


@pytest.mark.parametrize("centre", [range(4), range(6), np.zeros((2, 3)), 1.0, "abc"])
def test_centres_refused(centre):
    g = _Calls()
    with pytest.raises((TypeError, ValueError, IndexError)):
        g.fetchOccupancyAround(centre, 1.0)
    assert g.centres is None
