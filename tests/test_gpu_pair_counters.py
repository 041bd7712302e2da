"""Pair counts of contexts smaller than the query's 256 counters: the counters are zero
whatever their memory held before.  Whole numbers, against the oracle."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

SPEED = (1.0, 1.6)


@pytest.fixture
def used_memory(msim):
    """Small device allocations that hand out memory with old contents, as a program's do
    that has run for a while: blocks of 2 KB filled, and all but a few given back."""
    msim.Simulation(msim.RoadMap.lattice(2, 5), 1).close()  # the device's context is current
    cu, blocks = ctypes.CDLL("libcuda.so.1"), []
    for _ in range(4096):
        at = ctypes.c_uint64()
        assert cu.cuMemAlloc_v2(ctypes.byref(at), ctypes.c_size_t(2048)) == 0
        assert cu.cuMemsetD32_v2(at, ctypes.c_uint(0x1234567), ctypes.c_size_t(512)) == 0
        blocks.append(at)
    assert cu.cuCtxSynchronize() == 0
    for at in [b for i, b in enumerate(blocks) if i % 64]:
        cu.cuMemFree_v2(at)
    yield
    for at in blocks[::64]:
        cu.cuMemFree_v2(at)


@pytest.mark.parametrize("n", [1, 2, 33, 127, 128, 129])
def test_small_context_in_used_memory(msim, orc, used_memory, n):
    road_map = msim.RoadMap.lattice(2, 5)
    with msim.Simulation(road_map, n, rng="pcg32", dt=0.1, radius=6.0, cap=4) as sim:
        sim.init_entities(2, placement="fraction", speed=SPEED)
        for t in range(4):
            sim.step(1, neighbours=True)
            want = orc.neighbours(sim.get_state()["pos"], 6.0, 4)[2]
            assert sim.collision_pairs() == want, f"at tick {t + 1}"
