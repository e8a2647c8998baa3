"""cublox_integrate_noalloc on maps whose voxels do not fill their last
32-voxel line (one voxel, less than a line, a line and more), with hit
counters that are aligned for the fold by lines and hit counters that are
not; the caller's log-odds bit for bit the oracle's, the caller's counters zero afterwards, and
nothing written past the arrays' ends."""
import ctypes

import numpy as np
import pytest

import cublox_b200 as C
import oracle as O
from tests.test_zz_no_alloc import MapView, _entry

pytestmark = pytest.mark.gpu

LO = C.yaml_log_odds()


@pytest.mark.parametrize("shift", [0, 1], ids=["aligned", "unaligned"])
@pytest.mark.parametrize("half", [(0, 0, 0), (1, 1, 1), (2, 1, 0), (3, 2, 1), (17, 20, 9), (40, 33, 14)])
def test_noalloc_partial_lines(half, shift):
    import torch

    fn, _ = _entry()
    v = int(np.prod(2 * np.array(half) + 1))
    rng = np.random.default_rng(v)
    s = np.float32([0.031, 0.052, 0.047])
    buf = [torch.zeros(v + 40, dtype=t, device="cuda") for t in (torch.float32, torch.int32, torch.int32)]
    at = (0, 0, shift)  # where the arrays start in their buffers
    for b, a in zip(buf, at):
        b[v + a:] = 7
        b[:a] = 7
    occ, cnt, hit = (b[a:] for b, a in zip(buf, at))
    view = MapView(occ.data_ptr(), cnt.data_ptr(), hit.data_ptr(), (ctypes.c_int * 3)(*half),
                   (ctypes.c_int * 3)(0, 0, 0), 0.1, 0, 5.0, *LO[:4])
    o = O.OracleGrid(half, 0.1, False, None)
    o.set_log_odds(*LO)
    o.set_max_range(5.0)
    for n in (1, 300, 5000):
        p = (s + rng.normal(size=(n, 3)) * np.float32([1.5, 1.5, 0.6])).astype(np.float32)
        d = torch.from_numpy(np.ascontiguousarray(p.T)).cuda()
        assert fn(ctypes.byref(view), d.data_ptr(), n, (ctypes.c_float * 3)(*s), None) == C.OK
        o.update(p, s)
        torch.cuda.synchronize()
        assert np.array_equal(occ[:v].cpu().numpy().view(np.uint32), o.occ().view(np.uint32))
        assert not cnt[:v].any() and not hit[:v].any()
    for b, a in zip(buf, at):
        assert (b[v + a:] == 7).all() and (b[:a] == 7).all()
