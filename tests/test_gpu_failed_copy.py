"""An output array that CUDA refuses to copy to (its two ends are page-locked, what lies
between them is not) is an error of that call alone: what runs next is not reported to have
failed."""
import ctypes
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_refused_copy_is_reported_once(msim):
    lib = importlib.import_module(f"{msim.__name__}._capi").lib
    n, piece = 65536, 1 << 16  # counts over four pieces, the first and the last page-locked
    road_map = msim.RoadMap.lattice(24, 2)
    raw = np.zeros(n + piece // 4, np.uint32)
    at = (-raw.ctypes.data % piece) // 4
    count = raw[at:at + n]
    cu = ctypes.CDLL("libcuda.so.1")
    ends = [ctypes.c_void_p(count.ctypes.data + k * piece) for k in (0, 3)]
    with msim.Simulation(road_map, n, rng="pcg32", dt=0.1, radius=1.0, cap=0) as sim:
        sim.init_entities(3, placement="fraction", speed=(1.0, 1.6))
        sim.step(1, neighbours=True)
        want = sim.get_neighbours()[0]
        for p in ends:
            assert cu.cuMemHostRegister_v2(p, ctypes.c_size_t(piece), 0) == 0
        try:
            rc = lib().msim_get_neighbours(sim._ctx, count.ctypes.data_as(ctypes.POINTER(ctypes.c_uint32)), None)
            assert rc in (0, 3)
            sim.step(1, neighbours=False)
            sim.sync()
        finally:
            for p in ends:
                assert cu.cuMemHostUnregister(p) == 0
        assert rc == 3 or np.array_equal(count, want)
        with msim.Simulation(road_map, n, rng="pcg32", dt=0.1, radius=1.0, cap=0) as other:
            other.init_entities(3, placement="fraction", speed=(1.0, 1.6))
            other.step(2, neighbours=False)
            a, b = sim.get_state(), other.get_state()
    assert all(np.array_equal(a[k].view(np.uint32), b[k].view(np.uint32)) for k in a)
