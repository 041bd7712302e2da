"""The counting index update against full radix sorts (index="full") and the oracle, every
tick: counts around a warp, a block and a scan tile; one tile, few keys and the full key
space; everyone on one key, in runs of equal keys and one entity per key; slots in
spatial order (after re-orderings) and in the caller's; host ticks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(a, b):
    ca, ia = a.get_neighbours()
    cb, ib = b.get_neighbours()
    assert np.array_equal(ca, cb) and np.array_equal(ia, ib)
    assert a.collision_pairs() == b.collision_pairs()
    return ca, ia


@pytest.mark.parametrize("n,spread,cell,radius", [
    (1, 50.0, 0.0, 2.0), (31, 50.0, 0.0, 2.0), (257, 900.0, 0.0, 4.0), (4097, 900.0, 5000.0, 0.3),
    (4096, 1e-3, 0.0, 1e-6), (12_289, 0.5, 0.0, 0.004), (30_011, 900.0, 0.0, 2.0), (30_011, 900.0, 12.5, 2.0),
])
@pytest.mark.parametrize("resort", [2, 1000])
def test_counting_update_matches_full_sort(msim, orc, n, spread, cell, radius, resort):
    road_map = msim.RoadMap.lattice(20, 6)
    rs = np.random.default_rng(n)
    pos = (450.0 + rs.uniform(-0.5, 0.5, (n, 2)) * spread).astype(np.float32)
    head = (rs.integers(0, road_map.num_roads, n) | (rs.integers(0, 2, n) << 31)).astype(np.uint32)
    rng = rs.integers(1, 2**32, (n, 4), dtype=np.uint64).astype(np.uint32)
    speed = (rs.uniform(0.0, 1.0, n) * min(10.0, 20.0 * radius)).astype(np.float32)
    kw = dict(rng="xorshift128", dt=0.1, radius=radius, cap=8, cell_size=cell, resort_interval=resort, reuse=False)
    with msim.Simulation(road_map, n, **kw) as a, msim.Simulation(road_map, n, index="full", **kw) as b:
        for sim in (a, b):
            sim.set_entities(pos, head, rng, speed)
        for _ in range(7):
            for sim in (a, b):
                sim.step(1, neighbours=True)
            count, idx = _same(a, b)
        st = a.get_state()
        ocount, oidx, _ = orc.neighbours(st["pos"], radius, 8)
        assert np.array_equal(count, ocount) and np.array_equal(idx, oidx)
        for sim in (a, b):
            sim.step(5, neighbours=True)
        _same(a, b)
        # host ticks keep the caller's order
        sa, sb = a.get_state(), b.get_state()
        for _ in range(3):
            ga, gb = a.tick_host(sa, with_idx=True), b.tick_host(sb, with_idx=True)
            for k in ga:
                assert np.array_equal(ga[k].view(np.uint32), gb[k].view(np.uint32)), k
            sa, sb = {**ga, "speed": sa["speed"]}, {**gb, "speed": sb["speed"]}
