"""Batched ensembles about the line between pieces taken in turn and by tickets, with fewer
and more pieces than warps: every instance as if it ran alone, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[1], [31, 33, 1000], [260_000, 5, 70_001]])
@pytest.mark.parametrize("entities_per_thread", [1, 4])
def test_turns_and_tickets_match_single_runs(msim, sizes, entities_per_thread):
    road_map = msim.RoadMap.lattice(24, 3)
    runs = [1, 3, 4, 12, 13, 1, 63, 64, 65]
    with msim.Batch([road_map] * len(sizes), sizes) as batch:
        batch.init_entities(range(len(sizes)))
        batch.set_schedule(256, [0], [entities_per_thread], [4096])
        sims = [msim.Simulation(road_map, n, rng="pcg32", dt=0.1, radius=1.0, cap=0) for n in sizes]
        for i, sim in enumerate(sims):
            sim.init_entities(i, placement="fraction", speed=(1.0, 1.6))
        for ticks in runs:
            batch.step(ticks)
            for i, sim in enumerate(sims):
                sim.step(ticks)
                got, want = batch.get_state(i), sim.get_state()
                for k in want:
                    assert np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32)), (i, ticks, k)
        for sim in sims:
            sim.close()


def test_schedule_without_memory_for_it(msim):
    """A schedule whose work list finds no memory is refused, and the one before it goes on."""
    road_map, n = msim.RoadMap.lattice(12, 3), 50_000
    with msim.Batch([road_map], [n]) as batch, msim.Simulation(road_map, n, rng="pcg32", dt=0.1, radius=1.0,
                                                               cap=0) as sim:
        batch.init_entities([5])
        sim.init_entities(5, placement="fraction", speed=(1.0, 1.6))
        before = batch.schedule()
        msim.lib().msim_debug_fail_device_alloc(0)
        try:
            with pytest.raises(msim.MsimError) as e:
                batch.set_schedule(256, [0], [1], [1])  # a piece per entity
        finally:
            msim.lib().msim_debug_fail_device_alloc(-1)
        assert e.value.code == 5 and batch.schedule() == before
        batch.step(7)
        sim.step(7)
        got, want = batch.get_state(0), sim.get_state()
        assert all(np.array_equal(got[k].view(np.uint32), want[k].view(np.uint32)) for k in want)
