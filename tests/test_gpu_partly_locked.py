"""Outputs of which the first and the last element, but not what lies between, are
page-locked: the kernels write no such array themselves.  The copy that stands in for them
either arrives whole or reports an error."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PIECE = 1 << 16


@pytest.mark.parametrize("locked", [[(0, 6)], [(0, 3), (3, 3)], [(0, 2), (4, 2)], [(0, 2)], [(4, 2)], []])
def test_outputs_locked_in_parts(msim, locked):
    n = 5 * PIECE // 8  # positions over five pieces and the front of the sixth
    road_map, words = msim.RoadMap.lattice(24, 2), 2 * n + 64
    raw = np.zeros(8 * PIECE // 4, np.uint32)
    at = (-raw.ctypes.data % PIECE) // 4
    block = raw[at:at + words]
    out = block[:2 * n].view(np.float32).reshape(n, 2)
    cu = ctypes.CDLL("libcuda.so.1")
    with msim.Simulation(road_map, n, rng="pcg32", dt=0.1, radius=1.0, cap=4) as sim:
        sim.init_entities(3, placement="fraction", speed=(1.0, 1.6))
        sim.step(2, neighbours=True)
        want = sim.get_state()["pos"]
        spans = [(raw.ctypes.data + 4 * at + a * PIECE, k * PIECE) for a, k in locked]
        for p, size in spans:
            assert cu.cuMemHostRegister_v2(ctypes.c_void_p(p), ctypes.c_size_t(size), 0) == 0
        try:
            try:
                sim.get_state(out={"pos": out})
                assert np.array_equal(out.view(np.uint32), want.view(np.uint32))
            except msim.MsimError as e:  # the copy's own rule on such arrays
                assert e.code == 3 and len(locked) and sum(k for _, k in locked) < 6
            assert (block[2 * n:] == 0).all()
        finally:
            sim.sync()
            for p, _ in spans:
                assert cu.cuMemHostUnregister(ctypes.c_void_p(p)) == 0
        assert np.array_equal(sim.get_state()["pos"].view(np.uint32), want.view(np.uint32))
