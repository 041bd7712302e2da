"""Read-backs into page-locked arrays (written by the export kernels below 65,537
entities), into pageable ones and into page-locked ones off the kernels' alignment: the
same values, and the words around them untouched."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GUARD = 0x5A5A5A5A


def _guarded(msim, words, shift):
    """A page-locked array of `words` 32-bit words, `shift` words into its buffer, with guards."""
    buf = msim.PinnedBuffer(words + shift + 8, np.uint32)
    buf.array[:] = GUARD
    return buf, buf.array[shift:shift + words]


def _untouched(buf, words, shift):
    return bool((buf.array[:shift] == GUARD).all() and (buf.array[shift + words:] == GUARD).all())


@pytest.mark.parametrize("n", [1, 257, 65_536, 65_537])
@pytest.mark.parametrize("shift", [0, 1, 2, 4])
@pytest.mark.parametrize("cap", [5, 16])
def test_page_locked_outputs_match_pageable(msim, n, shift, cap):
    road_map = msim.RoadMap.lattice(12, 2)
    L, u32p, f32p = msim.lib(), ctypes.POINTER(ctypes.c_uint32), ctypes.POINTER(ctypes.c_float)
    with msim.Simulation(road_map, n, rng="pcg32", dt=0.1, radius=0.5, cap=cap) as sim:
        sim.init_entities(3, placement="fraction", speed=(1.0, 1.6))
        sim.step(2, neighbours=True)
        ref = sim.get_state()
        count, idx = sim.get_neighbours()
        sizes = {"pos": 2 * n, "heading": n, "rng": 4 * n, "speed": n, "count": n, "idx": n * cap}
        bufs = {k: _guarded(msim, w, shift) for k, w in sizes.items()}
        p = {k: b[1].ctypes.data for k, b in bufs.items()}
        msim.check(L.msim_get_state(sim._ctx, ctypes.cast(p["pos"], f32p), ctypes.cast(p["heading"], u32p),
                                    ctypes.cast(p["rng"], u32p), ctypes.cast(p["speed"], f32p)))
        msim.check(L.msim_get_neighbours(sim._ctx, ctypes.cast(p["count"], u32p), ctypes.cast(p["idx"], u32p)))
        want = {**{k: v.view(np.uint32).reshape(-1) for k, v in ref.items()}, "count": count, "idx": idx.reshape(-1)}
        for k, (buf, got) in bufs.items():
            assert np.array_equal(got, want[k]), k
            assert _untouched(buf, sizes[k], shift), k
        # single outputs
        bufs["pos"][1][:] = 0
        msim.check(L.msim_get_state(sim._ctx, ctypes.cast(p["pos"], f32p), None, None, None))
        assert np.array_equal(bufs["pos"][1], want["pos"])
