"""Memory of the pair lists: places by need in a large crowd, and an allocation that fails
once and is not tried again; counts, lists and pair counts against a context that updates
its index every tick."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(a, b):
    for x, y in zip(a.get_neighbours(), b.get_neighbours()):
        assert np.array_equal(x, y)
    assert a.collision_pairs() == b.collision_pairs()


def test_places_by_need(msim):
    """3 M entities with about 8 neighbours along the road: 93,750 warps, whose 3,072 places
    each would take 1.15 GB; with 1,024 384 MB beside 20 B per entity of other buffers."""
    road_map = msim.RoadMap.lattice(200, 5)
    kw = dict(rng="pcg32", dt=0.1, radius=4.8, cap=4)
    with msim.Simulation(road_map, 3_000_000, **kw) as a, msim.Simulation(road_map, 3_000_000, reuse=False, **kw) as b:
        before = a.info()["device_bytes"]
        for sim in (a, b):
            sim.init_entities(7, placement="fraction", speed=(1.0, 1.6))
        for _ in range(6):
            for sim in (a, b):
                sim.step(1, neighbours=True)
        _same(a, b)
        grown = a.info()["device_bytes"] - before
        assert 100e6 < grown < 600e6, grown


def test_no_memory_for_pair_lists(msim):
    road_map = msim.RoadMap.lattice(48, 5)
    kw = dict(rng="pcg32", dt=0.1, radius=2.0, cap=16)
    with msim.Simulation(road_map, 20_001, **kw) as a, msim.Simulation(road_map, 20_001, reuse=False, **kw) as b:
        for sim in (a, b):
            sim.init_entities(7, placement="fraction", speed=(1.0, 1.6))
        msim.lib().msim_debug_fail_device_alloc(1)  # the index reuse's buffers, not the pair lists'
        try:
            for sim in (a, b):
                sim.step(3, neighbours=True)
        finally:
            msim.lib().msim_debug_fail_device_alloc(-1)
        _same(a, b)
        size = a.info()["device_bytes"]
        for _ in range(30):
            for sim in (a, b):
                sim.step(1, neighbours=True)
        _same(a, b)
        assert a.info()["device_bytes"] == size
        assert a.sort_stats()["index_updates"] < b.sort_stats()["index_updates"]
