"""Read-backs above 65,536 entities: the state and id lists of 64 ids and more go straight
into page-locked arrays, counts and shorter lists through a copy; off the kernels'
alignment everything is copied.  The same values as pageable arrays hold, and the words
around them untouched."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GUARD = 0x5A5A5A5A


@pytest.mark.parametrize("n,cap", [(65_537, 63), (65_537, 64), (70_001, 67), (131_075, 64)])
@pytest.mark.parametrize("shift", [0, 1, 4])
def test_large_read_backs_match_pageable(msim, n, cap, shift):
    road_map = msim.RoadMap.lattice(24, 2)
    L, u32p, f32p = msim.lib(), ctypes.POINTER(ctypes.c_uint32), ctypes.POINTER(ctypes.c_float)
    with msim.Simulation(road_map, n, rng="xorshift128", dt=0.1, radius=1.0, cap=cap) as sim:
        sim.init_entities(3, placement="fraction", speed=(1.0, 1.6))
        sim.step(3, neighbours=True)
        ref = sim.get_state()
        count, idx = sim.get_neighbours()
        assert count.max() > 0
        want = {**{k: v.view(np.uint32).reshape(-1) for k, v in ref.items()}, "count": count, "idx": idx.reshape(-1)}
        bufs, p = {}, {}
        for k, v in want.items():
            bufs[k] = msim.PinnedBuffer(v.size + shift + 8, np.uint32)
            bufs[k].array[:] = GUARD
            p[k] = bufs[k].array[shift:].ctypes.data
        msim.check(L.msim_get_state(sim._ctx, ctypes.cast(p["pos"], f32p), ctypes.cast(p["heading"], u32p),
                                    ctypes.cast(p["rng"], u32p), ctypes.cast(p["speed"], f32p)))
        msim.check(L.msim_get_neighbours(sim._ctx, ctypes.cast(p["count"], u32p), ctypes.cast(p["idx"], u32p)))
        for k, v in want.items():
            got = bufs[k].array
            assert np.array_equal(got[shift:shift + v.size], v), k
            assert (got[:shift] == GUARD).all() and (got[shift + v.size:] == GUARD).all(), k
            bufs[k].free()
