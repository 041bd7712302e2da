"""Id lists longer than a query kernel keeps per entity (32 in the dense one, 48 in the
one for crowds), rebuilt from the warp's pairs by the query that keeps them and by those
that read them: counts around both, warps whose lists fit the kept words at once, in
groups of lanes, or not at all, and caps below, at and above.  Integers, so equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RADIUS, WORLD = 4.0, 2000.0
SIZES = [32, 33, 34, 35, 48, 49, 50, 51, 65, 97, 130, 300, 1600] + [33, 36, 50, 3, 1] * 12


def _clusters(seed):
    rs = np.random.default_rng(seed)
    side = int(np.ceil(np.sqrt(len(SIZES))))
    pitch = WORLD / side
    pos = [np.array([(k % side + 0.5) * pitch, (k // side + 0.5) * pitch]) + rs.uniform(-0.3, 0.3, (m, 2)) * RADIUS
           for k, m in enumerate(SIZES)]  # all within 0.85 radius of each other
    pos = np.concatenate(pos).astype(np.float32)
    return pos[rs.permutation(pos.shape[0])]


@pytest.mark.parametrize("expected", [0.6, 3.0, 20.0])  # neighbours along the road: picks the kernel
@pytest.mark.parametrize("cap", [0, 1, 33, 49, 64, 256])
def test_long_lists_match_oracle(msim, orc, expected, cap):
    pos = _clusters(cap)
    n = pos.shape[0]
    length = 2.0 * RADIUS * n / expected
    road_map = msim.RoadMap(np.float32([[0.0, 0.0, length, 1.0]]), np.zeros((1, 4), np.uint32),
                            np.zeros(0, np.uint32), WORLD, WORLD)
    head = np.full(n, 0x80000000, np.uint32)
    rng = np.ones((n, 4), np.uint32)
    speed = np.random.default_rng(1).uniform(0.2, 1.0, n).astype(np.float32)
    with msim.Simulation(road_map, n, rng="pcg32", dt=0.05, radius=RADIUS, cap=cap) as sim:
        sim.set_entities(pos, head, rng, speed)
        ticks = 24
        for tick in range(ticks):
            sim.step(1, neighbours=True)
            orc.step(road_map.road_pos, road_map.road_conn, road_map.connections, pos, head, rng, speed, 1, 0.05, 1)
            count, idx = sim.get_neighbours()
            ref_count, ref_idx, _ = orc.neighbours(pos, RADIUS, cap, with_idx=cap > 0)
            assert np.array_equal(count, ref_count), f"counts differ at tick {tick + 1}"
            assert cap == 0 or np.array_equal(idx, ref_idx), f"lists differ at tick {tick + 1}"
        assert sim.sort_stats()["index_updates"] < ticks  # so lists were kept and read back
