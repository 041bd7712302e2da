"""Pair lists of the ticks that reuse an index, against a context that updates its
index every tick: counts, id lists and pair counts of every tick.  Sparse and dense
kernels, warps whose pairs do not fit their places (they look them up), lists kept
again inside a reuse window, one entity and counts around a warp and a block,
move-only ticks in between, factors set in between, entities of speed zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _compare(a, b):
    ca, ia = a.get_neighbours()
    cb, ib = b.get_neighbours()
    assert np.array_equal(ca, cb)
    assert (ia is None and ib is None) or np.array_equal(ia, ib)
    assert a.collision_pairs() == b.collision_pairs()
    return ca


@pytest.mark.parametrize("n,side,radius,speed,dt,cap,rng", [
    (1, 4, 2.0, (1.0, 1.6), 0.1, 4, "pcg32"),
    (31, 4, 2.0, (1.0, 1.6), 0.1, 4, "pcg32"),
    (129, 4, 3.0, (0.0, 0.0), 0.1, 16, "xorshift128"),
    (20_001, 48, 2.0, (1.0, 1.6), 0.1, 64, "pcg32"),       # sparse, a dozen ticks a window
    (20_001, 48, 2.0, (0.1, 0.2), 0.1, 8, "xorshift128"),  # sparse, lists kept again in a window
    (30_000, 24, 1.2, (1.0, 1.6), 0.05, 64, "pcg32"),      # about the border of the kernels
    (30_000, 24, 10.0, (1.4, 1.4), 1.0, 64, "xorshift128"),  # dense, long steps
    (30_000, 12, 6.0, (1.0, 1.6), 0.1, 16, "pcg32"),       # dense, places overflow
    (9_000, 48, 2.0, (1.0, 1.6), 0.1, 0, "pcg32"),         # counts only
])
def test_pair_lists_match_updates_every_tick(msim, n, side, radius, speed, dt, cap, rng):
    road_map = msim.RoadMap.lattice(side, 5)
    rs = np.random.default_rng(n)
    kw = dict(rng=rng, dt=dt, radius=radius, cap=cap)
    with msim.Simulation(road_map, n, **kw) as a, msim.Simulation(road_map, n, reuse=False, **kw) as b:
        for sim in (a, b):
            sim.init_entities(7, placement="fraction", speed=speed)
        total = 0
        for tick in range(70):
            for sim in (a, b):
                sim.step(1, neighbours=True)
            total += int(_compare(a, b).sum())
            if tick in (20, 33):  # move-only ticks inside a window
                for sim in (a, b):
                    sim.step(2)
            if tick == 45:  # a new bound
                f = rs.uniform(0.5, 1.5, road_map.num_roads).astype(np.float32)
                for sim in (a, b):
                    sim.set_road_factors(f)
        assert n < 1000 or total > 0
        for sim in (a, b):  # several ticks a call: the queries overlap the next moves
            sim.step(9, neighbours=True)
        _compare(a, b)
        assert a.sort_stats()["index_updates"] < b.sort_stats()["index_updates"]


@pytest.mark.parametrize("radius", [1.0, 8.0])
def test_clusters_beyond_the_places(msim, radius):
    """Clusters of up to 3,000 entities: a warp's pairs pass its places by far."""
    rs = np.random.default_rng(1)
    sizes = [3000, 400, 100, 40] + [1] * 3000
    pos = np.concatenate([rs.uniform(100, 1900, 2) + rs.normal(0, 0.5 * radius, (m, 2)) for m in sizes])
    pos = np.clip(pos, 0.5, 1999.0).astype(np.float32)
    n = pos.shape[0]
    road_map = msim.RoadMap(np.float32([[0.0, 0.0, 2000.0, 2000.0]]), np.zeros((1, 4), np.uint32),
                            np.zeros(0, np.uint32), 2000.0, 2000.0)
    head = np.full(n, 0x80000000, np.uint32)
    speed = rs.uniform(0.0, 1.0, n).astype(np.float32)
    kw = dict(rng="pcg32", dt=0.05, radius=radius, cap=32)
    with msim.Simulation(road_map, n, **kw) as a, msim.Simulation(road_map, n, reuse=False, **kw) as b:
        for sim in (a, b):
            sim.set_entities(pos, head, np.ones((n, 4), np.uint32), speed)
        for _ in range(40):
            for sim in (a, b):
                sim.step(1, neighbours=True)
            _compare(a, b)
