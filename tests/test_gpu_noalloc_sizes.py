"""The allocation-free neighbour query over its sizes and forms: one entity to the
limit, worlds of one cell, thin and square, radii from zero to the whole world, caps
with and without 16-byte rows, an id output off a 16-byte boundary, positions outside
the world and not finite; counts and ids equal to the oracle's."""
import ctypes
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _call(msim, torch, pos, w, h, radius, cap, offset=0):
    fn = msim.lib().msim_query_neighbours_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_void_p, ctypes.c_uint32, ctypes.c_float, ctypes.c_float, ctypes.c_float, ctypes.c_uint32,
                   ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    n = pos.shape[0]
    d_pos = torch.from_numpy(pos).cuda()
    count = torch.full((n,), -2, dtype=torch.int32, device="cuda")
    idx = torch.full((n * max(cap, 1) + offset,), -2, dtype=torch.int32, device="cuda")
    status = torch.full((1,), 7, dtype=torch.int32, device="cuda")
    rc = fn(d_pos.data_ptr(), n, w, h, radius, cap, count.data_ptr(), idx[offset:].data_ptr() if cap else None,
            status.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert rc == 0, msim.lib().msim_last_error()
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    return count.cpu().numpy().view(np.uint32), idx[offset:].cpu().numpy().view(np.uint32).reshape(n, -1)[:, :cap]


@pytest.mark.parametrize("n,w,h,radius,cap,offset", [
    (1, 10.0, 10.0, 2.0, 4, 0), (2, 0.5, 0.5, 2.0, 1, 0), (127, 50.0, 40.0, 0.0, 8, 0), (129, 1e5, 3.0, 5.0, 7, 0),
    (1000, 3.0, 4e4, 20.0, 16, 1), (1025, 100.0, 100.0, 500.0, 256, 0), (5000, 300.0, 200.0, 3.0, 0, 0),
    (20_001, 2000.0, 1500.0, 4.0, 12, 2), (100_003, 4000.0, 4000.0, 2.0, 16, 0), (262_144, 3000.0, 3000.0, 3.0, 5, 0),
])
def test_sizes_match_oracle(msim, orc, n, w, h, radius, cap, offset):
    torch = pytest.importorskip("torch")
    rs = np.random.default_rng(n)
    pos = rs.uniform([0, 0], [w, h], (n, 2)).astype(np.float32)
    if n > 100:  # a cluster, equal positions, and positions outside the world
        k = n // 10
        pos[:k] = (pos[0] + rs.normal(0, radius + 0.1, (k, 2))).astype(np.float32)
        pos[k:k + 20] = pos[k]
        pos[k + 20:k + 40] *= np.float32(3.0)
        pos[k + 40:k + 50] *= np.float32(-1.0)
    for _ in range(2):  # the second call finds the first one's scratch
        count, idx = _call(msim, torch, pos, w, h, radius, cap, offset)
        ocount, oidx, _ = orc.neighbours(pos, radius, cap)
        assert np.array_equal(count, ocount)
        if cap:
            assert np.array_equal(idx, oidx)


def test_not_finite_positions_have_no_neighbours(msim, orc):
    torch = pytest.importorskip("torch")
    rs = np.random.default_rng(4)
    pos = rs.uniform(0, 60, (3000, 2)).astype(np.float32)
    pos[::50, 0] = np.nan
    pos[1::50] = np.inf
    pos[2::50, 1] = -np.inf
    count, idx = _call(msim, torch, pos, 60.0, 60.0, 3.0, 32)
    fine = np.isfinite(pos).all(1)
    assert not count[~fine].any()
    ids = np.nonzero(fine)[0]
    ocount, oidx, _ = orc.neighbours(pos[fine], 3.0, 32)
    assert np.array_equal(count[fine], ocount)
    want = np.where(oidx == 0xFFFFFFFF, 0xFFFFFFFF, ids[np.minimum(oidx, ids.size - 1)])
    assert np.array_equal(idx[fine], want)
