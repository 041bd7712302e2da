"""A host tick that is refused for an invalid heading leaves nothing behind that the ticks
after it count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPEED = (1.0, 1.6)


def _arrays(msim, st, n, pinned):
    """The state and a count array, page-locked or not, and what keeps them alive."""
    shapes = {k: (v.shape, v.dtype) for k, v in st.items()} | {"count": ((n,), np.dtype(np.uint32))}
    bufs = {k: msim.PinnedBuffer(*s) for k, s in shapes.items()} if pinned else {}
    state = {k: bufs[k].array if pinned else np.empty(*s) for k, s in shapes.items()}
    for k in st:
        state[k][...] = st[k]
    return bufs, state


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("moved", [3.0, np.nan])
def test_refused_host_tick_leaves_no_counts(msim, pinned, moved):
    """A host tick with an invalid heading and entities further than the radius from where
    they were (or nowhere): refused, and the next ticks count their own pairs."""
    road_map = msim.RoadMap.lattice(16, 2)
    n = 30_001
    kw = dict(rng="pcg32", dt=0.1, radius=2.0, cap=4)
    with msim.Simulation(road_map, n, **kw) as a, msim.Simulation(road_map, n, **kw) as b:
        a.init_entities(1, placement="fraction", speed=SPEED)
        bufs, state = _arrays(msim, a.get_state(), n, pinned)
        for _ in range(3):
            a.tick_host(state, neighbours=True, out=state)
        before = {k: state[k].copy() for k in ("pos", "heading", "rng")}
        state["pos"][::5] += np.float32(moved)
        state["heading"][77] = road_map.num_roads
        with pytest.raises(msim.MsimError) as e:
            a.tick_host(state, neighbours=True, out=state)
        assert e.value.code == 2
        for k in before:
            state[k][...] = before[k]
        b.set_entities(state["pos"], state["heading"], state["rng"], state["speed"])
        for t in range(4):
            if t < 2:
                a.tick_host(state, neighbours=True, out=state)
            else:
                a.step(1, neighbours=True)
            b.step(1, neighbours=True)
            assert a.collision_pairs() == b.collision_pairs(), f"at tick {t + 1}"
        for buf in bufs.values():
            buf.free()


def test_time_out_before_a_refused_host_tick(msim, orc):
    """Refused while the index update that the call before left running had given up: the
    key counters are zeroed before they count again, so the ticks after it match the oracle
    (whole numbers and the same binary32 operations)."""
    rm = msim.RoadMap.lattice(32, 3)
    n, cap = 150_000, 8
    pos, head, rng, speed = orc.init_entities(rm.road_pos, n, 1, 11, 1, 1.0, 1.6)
    with msim.Simulation(rm, n, rng="pcg32", dt=0.1, radius=2.0, cap=cap) as sim:
        state = {"pos": pos.copy(), "heading": head.copy(), "rng": rng.copy(), "speed": speed}

        def host_tick(what):
            nonlocal state
            got = sim.tick_host(state, neighbours=True, with_idx=True)
            orc.step(rm.road_pos, rm.road_conn, rm.connections, pos, head, rng, speed, 1, 0.1, 1, threads=8)
            assert np.array_equal(got["pos"].view(np.uint32), pos.view(np.uint32)), what
            count, idx, pairs = orc.neighbours(pos, 2.0, cap, threads=8)
            assert np.array_equal(got["count"], count) and np.array_equal(got["idx"], idx), what
            assert sim.collision_pairs() == pairs, what
            state = {"pos": got["pos"].copy(), "heading": got["heading"].copy(), "rng": got["rng"].copy(),
                     "speed": speed}

        for t in range(2):
            host_tick(f"tick {t + 1}")
        sim.set_wait_limit(2048)
        sim.inject_fault(msim._capi.FAULT_SORT_TILE)  # the update after this tick's query gives up
        state = sim.tick_host(state, neighbours=True) | {"speed": speed}
        orc.step(rm.road_pos, rm.road_conn, rm.connections, pos, head, rng, speed, 1, 0.1, 1, threads=8)
        bad = {k: v.copy() for k, v in state.items()}
        bad["heading"][3] = rm.num_roads
        with pytest.raises(msim.MsimError) as e:
            sim.tick_host(bad, neighbours=True)
        assert e.value.code == 2
        sim.set_wait_limit(0)
        state = {k: state[k] for k in ("pos", "heading", "rng", "speed")}
        for t in range(5):
            host_tick(f"tick {t + 1} after the refusal")
        sim.sync()
