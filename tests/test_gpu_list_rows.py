"""Neighbour read-backs about the lines of their writers: lists written end to end, entity
after entity and 16 bytes a lane, in place or staged; page-locked and pageable arrays hold
the same whole numbers, and the words behind them stay."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 12_288, 12_289, 32_768, 32_769])
@pytest.mark.parametrize("cap", [1, 2, 3, 4, 22, 23, 24, 25, 32, 33, 96])
def test_lists_about_their_writers_lines(msim, orc, n, cap):
    road_map = msim.RoadMap.lattice(max(4, int((n / 40) ** 0.5)), 2)
    with msim.Simulation(road_map, n, rng="pcg32", dt=0.1, radius=4.0, cap=cap) as sim:
        sim.init_entities(3, placement="fraction", speed=(1.0, 1.6))
        sim.step(2, neighbours=True)
        count, idx, _ = orc.neighbours(sim.get_state()["pos"], 4.0, cap, threads=8)
        assert np.array_equal(sim.get_neighbours(with_idx=False)[0], count)
        bufs = [msim.PinnedBuffer(n + 8, np.uint32), msim.PinnedBuffer(n * cap + 8, np.uint32)]
        for b in bufs:
            b.array[:] = 0x5A5A5A5A
        out = bufs[0].array[:n], bufs[1].array[: n * cap].reshape(n, cap)
        sim.get_neighbours(out=out)
        assert np.array_equal(out[0], count) and np.array_equal(out[1], idx)
        assert all(np.array_equal(a, b) for a, b in zip(sim.get_neighbours(), (count, idx)))
        assert all((b.array[-8:] == 0x5A5A5A5A).all() for b in bufs)
        for b in bufs:
            b.free()
