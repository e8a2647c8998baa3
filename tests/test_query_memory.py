"""query_states on points and states in every kind of memory, and on pinned
points that the grid's stream is still to write."""
import ctypes

import numpy as np
import pytest

import cublox_b200 as C

pytestmark = pytest.mark.gpu


def _grid(stream=None):
    half = (20, 20, 8)
    g = C.OccupancyGrid(half, 0.1, False, None, stream=stream)
    g.import_(np.random.default_rng(1).choice(np.float32([-1, 0, 2]), int(np.prod(2 * np.array(half) + 1))))
    return g


def _query(g, xyz, n, out):
    rc = C.lib().cublox_grid_query_states(g._h, ctypes.cast(xyz, ctypes.POINTER(ctypes.c_float)), n,
                                          ctypes.cast(out, ctypes.POINTER(ctypes.c_uint8)))
    assert rc == C.OK, C.lib().cublox_last_error()


@pytest.mark.parametrize("n", [1, 129, 70000])
@pytest.mark.parametrize("points", ["pageable", "pinned", "device"])
@pytest.mark.parametrize("states", ["pageable", "pinned", "device"])
def test_kinds_of_memory(n, points, states):
    import torch

    def of(kind, t):
        return t.cuda() if kind == "device" else (t.pin_memory() if kind == "pinned" else t)

    g = _grid()
    p = torch.from_numpy(np.random.default_rng(n).uniform(-2.5, 2.5, (n, 3)).astype(np.float32))
    want = g.query_states(p.numpy())
    assert n == 1 or set(want) == {0, 1, 2}
    x, out = of(points, p), of(states, torch.full((n,), 9, dtype=torch.uint8))
    torch.cuda.synchronize()
    _query(g, x.data_ptr(), n, out.data_ptr())
    assert np.array_equal(out.cpu().numpy(), want)
    assert np.array_equal(x.cpu().numpy(), p.numpy())
    g.close()


@pytest.mark.parametrize("n", [256, 70000])
def test_pinned_points_written_by_earlier_work_of_the_stream(n):
    """A copy into the pinned points that is queued on the grid's stream, behind
    milliseconds of work, comes before the query that is queued after it."""
    import torch

    st = torch.cuda.Stream()
    g = _grid(st.cuda_stream)
    p = np.random.default_rng(n).uniform(-2.0, 2.0, (n, 3)).astype(np.float32)
    want = g.query_states(p)
    out = np.zeros(n, np.uint8)
    x = torch.full((n, 3), 100.0).pin_memory()  # outside the window: all unknown
    d = torch.from_numpy(p).cuda()
    a = torch.randn(4096, 4096, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        for _ in range(20):
            a = a @ a * 1e-3
        x.copy_(d, non_blocking=True)
        _query(g, x.data_ptr(), n, out.ctypes.data)
    assert np.array_equal(out, want)
    g.close()
