"""Neighbour counts and id lists around the sizes where the query's list code changes
path: lists kept in registers (8), kept in shared memory (32 in the dense kernel),
collected by the warp (32 words per kept place: 256 and 1,024) and inserted by a lane
(beyond), for caps below, at and above them, in both kernels; integers, so equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# clusters of these sizes: every member has size - 1 neighbours
SIZES = [1, 2, 3, 8, 9, 10, 16, 31, 32, 33, 34, 65, 120, 256, 257, 258, 300, 1024, 1025, 1030]


def _clusters(seed, radius, world):
    rs = np.random.default_rng(seed)
    sizes = np.array(SIZES + [1, 2, 9, 12, 20, 33] * 20)
    side = int(np.ceil(np.sqrt(sizes.size)))
    pitch = world / side
    pos = []
    for k, m in enumerate(sizes):
        centre = np.array([(k % side + 0.5) * pitch, (k // side + 0.5) * pitch])
        pos.append(centre + rs.uniform(-0.3, 0.3, (m, 2)) * radius)  # all within 0.85 radius of each other
    pos = np.concatenate(pos).astype(np.float32)
    return pos[rs.permutation(pos.shape[0])]


@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("cap", [0, 1, 7, 8, 9, 31, 33, 64, 256])
@pytest.mark.parametrize("cell", [0.0, 9.0])  # automatic tiles; boxes over three tiles and more
def test_lists_match_oracle(msim, orc, dense, cap, cell):
    radius, world = 4.0, 2000.0
    pos = _clusters(cap, radius, world)
    n = pos.shape[0]
    # road length sets the expected density: n entities x 8 m against 1.5 per entity
    length = 0.5 * world if dense else 2000.0 * world
    road = np.float32([[0.0, 0.0, length, 1.0]])
    road_map = msim.RoadMap(road, np.zeros((1, 4), np.uint32), np.zeros(0, np.uint32), world, world)
    with msim.Simulation(road_map, n, dt=1.0, radius=radius, cap=cap, cell_size=cell) as sim:
        sim.set_entities(pos, np.full(n, 0x80000000, np.uint32), np.ones((n, 4), np.uint32), np.zeros(n, np.float32))
        for _ in range(3):  # the full sort, an update or reuse after it, and once more
            sim.step(1, neighbours=True)
        assert np.array_equal(sim.get_state()["pos"], pos)
        count, idx = sim.get_neighbours()
        pairs = sim.collision_pairs()
    ocount, oidx, opairs = orc.neighbours(pos, radius, cap)
    assert np.array_equal(count, ocount) and pairs == int(ocount.sum()) // 2
    if cap:
        assert np.array_equal(idx, oidx)
