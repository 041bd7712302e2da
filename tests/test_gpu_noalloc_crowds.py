"""The no-allocation query over crowds, against the oracle (whole numbers): lists of no, a
few, 32 and 33, 64 and 65, and the most ids; shorter and longer than the neighbours there
are; ids in no order; small grids whose chain runs on few SMs."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [2, 30, 33, 34, 60, 64, 65, 66, 100, 255, 256, 257, 258, 700, 1500]  # all in range of each other


@pytest.mark.parametrize("cap", [0, 1, 4, 31, 32, 33, 64, 65, 100, 200, 256])
@pytest.mark.parametrize("world", [300.0, 4000.0])
def test_crowds(msim, orc, cap, world):
    torch = pytest.importorskip("torch")
    fn = msim.lib().msim_query_neighbours_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_void_p, ctypes.c_uint32, ctypes.c_float, ctypes.c_float, ctypes.c_float, ctypes.c_uint32,
                   ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    rs = np.random.default_rng(cap)
    pos = [rs.uniform(0.05, 0.95, 2) * world + rs.uniform(-0.6, 0.6, (m, 2)) for m in SIZES]
    pos = np.concatenate(pos + [rs.uniform(0, world, (1000, 2))]).astype(np.float32)
    pos = pos[rs.permutation(len(pos))]
    n = len(pos)
    d_pos = torch.from_numpy(pos).cuda()
    count = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    idx = torch.full((n, max(cap, 1)), -2, dtype=torch.int32, device="cuda")
    for _ in range(2):
        assert fn(d_pos.data_ptr(), n, world, world, 2.0, cap, count.data_ptr(), idx.data_ptr() if cap else None, None,
                  torch.cuda.current_stream().cuda_stream) == 0
    want, ids, _ = orc.neighbours(pos, 2.0, cap, threads=8)
    assert want.max() >= 1499
    assert np.array_equal(count.cpu().numpy().view(np.uint32), want)
    if cap:
        assert np.array_equal(idx.cpu().numpy().view(np.uint32), ids)
