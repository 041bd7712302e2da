"""Id lists of entities with more neighbours than a query keeps, against the oracle (whole
numbers): clusters whose lists fit the warp's words at once, in two turns, not at all; that
pass the words by far; many and few of them in a warp; every query kernel (by the road's
length), looked up, kept and read back (ticks that reuse the index)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# entities of a cluster, all within reach of each other: a list of one less
SIZES = [9, 10, 21, 22, 34, 41, 42, 50, 65, 97, 98, 130, 260, 400, 650, 1300, 2100]


def _population(radius, seed):
    rs = np.random.default_rng(seed)
    pos = [rs.uniform(50, 1900, 2) + rs.uniform(-0.3, 0.3, (m, 2)) * radius for m in SIZES for _ in range(1 + 60 // m)]
    pos = np.concatenate(pos + [rs.uniform(1, 1999, (1500, 2))]).astype(np.float32)
    return pos[rs.permutation(len(pos))]  # ids in no order


@pytest.mark.parametrize("radius", [0.1, 0.4, 2.0])  # neighbours along the road: 0.6, 2.4, 12
@pytest.mark.parametrize("cap", [1, 8, 16, 20, 33, 64, 96, 100, 256])
def test_lists_beyond_the_kept_places(msim, orc, radius, cap):
    pos = _population(radius, cap)
    n = len(pos)
    road_map = msim.RoadMap(np.float32([[0.0, 0.0, 2000.0, 2000.0]]), np.zeros((1, 4), np.uint32),
                            np.zeros(0, np.uint32), 2000.0, 2000.0)
    rs = np.random.default_rng(1)
    speed = (rs.uniform(0.0, 0.02, n) * radius).astype(np.float32)
    with msim.Simulation(road_map, n, rng="pcg32", dt=1.0, radius=radius, cap=cap) as sim:
        sim.set_entities(pos, np.full(n, 0x80000000, np.uint32), np.ones((n, 4), np.uint32), speed)
        for t in range(4):
            sim.step(1, neighbours=True)
            count, idx, pairs = orc.neighbours(sim.get_state()["pos"], radius, cap, threads=8)
            got, ids = sim.get_neighbours()
            assert count.max() > 2000
            assert np.array_equal(got, count) and np.array_equal(ids, idx), f"at tick {t + 1}"
            assert sim.collision_pairs() == pairs
