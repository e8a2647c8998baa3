"""cublox_integrate_noalloc on arrays that start off a 16-byte boundary: the
log-odds bit for bit the oracle's, the counters zero afterwards and nothing
written around the arrays, for every place in a 16-byte group at which the
stored values and counters may start, on maps of fewer voxels than the ones
before the first aligned counter and of more.  Arrays off a 4-byte boundary
are refused on the host."""
import ctypes

import numpy as np
import pytest

import cublox_b200 as C
import oracle as O
from tests.test_zz_no_alloc import MapView, _entry

LO = C.yaml_log_odds()


@pytest.mark.gpu
@pytest.mark.parametrize("at", [(1, 0, 0), (0, 1, 0), (0, 2, 1), (2, 3, 0), (3, 3, 3)], ids=str)
@pytest.mark.parametrize("half", [(0, 0, 0), (1, 0, 0), (2, 1, 0), (17, 20, 9)], ids=str)
def test_noalloc_unaligned_arrays(half, at):
    import torch

    fn, _ = _entry()
    v = int(np.prod(2 * np.array(half) + 1))
    rng = np.random.default_rng(v)
    s = np.float32([0.031, 0.052, 0.047])
    buf = [torch.zeros(v + 40, dtype=t, device="cuda") for t in (torch.float32, torch.int32, torch.int32)]
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
        p[0] = s + np.float32([0.01, 0.01, 0.01])  # a hit in the sensor's own voxel
        d = torch.from_numpy(np.ascontiguousarray(p.T)).cuda()
        assert fn(ctypes.byref(view), d.data_ptr(), n, (ctypes.c_float * 3)(*s), None) == C.OK
        o.update(p, s)
        torch.cuda.synchronize()
        assert np.array_equal(occ[:v].cpu().numpy().view(np.uint32), o.occ().view(np.uint32))
        assert not cnt[:v].any() and not hit[:v].any()
    for b, a in zip(buf, at):
        assert (b[v + a:] == 7).all() and (b[:a] == 7).all()


@pytest.mark.parametrize("which", range(4), ids=["occ", "cnt", "hit", "points"])
@pytest.mark.parametrize("off", [1, 2, 3])
def test_noalloc_refuses_arrays_off_a_4_byte_boundary(which, off):
    fn, L = _entry()
    ptr = [1 << 20, 1 << 21, 1 << 22, 1 << 23]  # never dereferenced: refused first
    ptr[which] += off
    view = MapView(*ptr[:3], (ctypes.c_int * 3)(4, 4, 4), (ctypes.c_int * 3)(0, 0, 0), 0.1, 0, 5.0, *LO[:4])
    so = (ctypes.c_float * 3)(0.0, 0.0, 0.0)
    assert fn(ctypes.byref(view), ptr[3], 8, so, None) == C.ERR_INVALID
    assert b"4-byte boundary" in L.cublox_noalloc_last_error()
