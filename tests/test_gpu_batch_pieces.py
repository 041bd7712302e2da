"""Batched ensemble at the sizes where its work is cut: instances of no, one, a warp's
and a warp's plus or minus one entities beside large ones, one, two and four entities a
thread, tick counts on both sides of the early RNG load; bit-identical to each alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [0, 1, 31, 32, 33, 127, 129, 4097, 60_001]


@pytest.mark.parametrize("rng", ["pcg32", "xorshift128"])
@pytest.mark.parametrize("per_thread,block", [(1, 256), (2, 96), (4, 512)])
def test_pieces_match_single_instances(msim, rng, per_thread, block):
    maps = [msim.RoadMap.lattice(8 + k, k) for k in range(len(SIZES))]
    seeds = list(range(100, 100 + len(SIZES)))
    runs = (1, 63, 64, 65)
    with msim.Batch(maps, SIZES, rng=rng, dt=0.5) as b:
        b.init_entities(seeds)
        b.set_schedule(block, [0], [per_thread], [5000])
        assert b.info()["work_items"] == sum(-(-n // 5000) for n in SIZES)
        for t in runs:
            b.step(t)
        states = [b.get_state(i) for i in range(len(SIZES))]
    for got, m, n, seed in zip(states, maps, SIZES, seeds):
        if n == 0:
            continue
        with msim.Simulation(m, n, rng=rng, dt=0.5, radius=2.0, cap=0) as sim:
            sim.init_entities(seed, placement="fraction", speed=(1.0, 1.6))
            sim.step(sum(runs))
            ref = sim.get_state()
        for k in ("pos", "heading", "rng", "speed"):
            assert np.array_equal(got[k].view(np.uint32), ref[k].view(np.uint32)), (n, k)
