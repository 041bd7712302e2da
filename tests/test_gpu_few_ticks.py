"""Runs of one to a few move ticks against the oracle, bit for bit: counts below and at a full
warp per 32 entities, and more entities than the grids of the fixed tick counts hold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 38_911, 38_912, 311_297, 940_001])
@pytest.mark.parametrize("rng", ["pcg32", "xorshift128"])
def test_few_ticks_match_the_oracle(msim, orc, n, rng):
    road_map = msim.RoadMap.lattice(40, 3)
    kind = {"xorshift128": 0, "pcg32": 1}[rng]
    pos, head, state, speed = orc.init_entities(road_map.road_pos, n, kind, 3, 1, 1.0, 1.6)
    with msim.Simulation(road_map, n, rng=rng, dt=2.0, radius=1.0, cap=0) as sim:
        sim.set_entities(pos, head, state, speed)
        for ticks in (1, 2, 3, 4, 5):
            sim.step(ticks)
            orc.step(road_map.road_pos, road_map.road_conn, road_map.connections, pos, head, state, speed, kind, 2.0,
                     ticks, threads=8)
            got = sim.get_state()
            assert np.array_equal(got["pos"].view(np.uint32), pos.view(np.uint32)), f"positions after {ticks} more"
            assert np.array_equal(got["heading"], head) and np.array_equal(got["rng"], state)
