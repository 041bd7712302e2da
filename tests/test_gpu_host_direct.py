"""Host ticks whose arrays are all page-locked and both input and output: one kernel reads
the state over the link, moves it and writes the results back.  Compared bit for bit with
the same tick through the separate calls (whole numbers and the same binary32 operations,
so no tolerance)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pinned(msim, st, n, speed):
    names = ("pos", "heading", "rng") + (("speed",) if speed else ())
    bufs = {k: msim.PinnedBuffer(st[k].shape, st[k].dtype) for k in names}
    bufs["count"] = msim.PinnedBuffer(n, np.uint32)
    state = {k: b.array for k, b in bufs.items()}
    for k in names:
        state[k][...] = st[k]
    return bufs, state


def _same(got, ref, cnt, what):
    assert np.array_equal(got["pos"].view(np.uint32), ref["pos"].view(np.uint32)), f"positions {what}"
    assert np.array_equal(got["heading"], ref["heading"]), f"headings {what}"
    assert np.array_equal(got["rng"], ref["rng"]), f"RNG states {what}"
    assert np.array_equal(got["count"], cnt), f"counts {what}"


# one entity; a block of the move kernel less and more one; more than its blocks hold at once
@pytest.mark.parametrize("n", [1, 511, 513, 70_001, 320_003])
@pytest.mark.parametrize("rng,speed", [("pcg32", True), ("xorshift128", False)])
def test_direct_host_ticks_match_separate_calls(msim, n, rng, speed):
    """Five ticks; before the fourth the host moves entities further than the radius, so
    that the previous index does not serve and the query runs on the new one."""
    road_map = msim.RoadMap.lattice(40, 3)
    kw = dict(rng=rng, dt=0.1, radius=2.0, cap=8)
    with msim.Simulation(road_map, n, **kw) as a, msim.Simulation(road_map, n, **kw) as b:
        a.init_entities(4, placement="fraction", speed=(1.0, 1.6) if speed else (1.4, 1.4))
        bufs, state = _pinned(msim, a.get_state(), n, speed)
        for t in range(5):
            if t == 3:
                state["pos"][::7] += np.float32(3.0)
            b.set_entities(state["pos"], state["heading"], state["rng"], state.get("speed"))
            b.step(1, neighbours=True)
            a.tick_host(state, neighbours=True, out=state)
            _same(state, b.get_state(), b.get_neighbours(with_idx=False)[0], f"at tick {t + 1}")
            assert a.collision_pairs() == b.collision_pairs()
            if t == 2:  # lists of the same query, and the context's own state
                ids, ref_ids = a.get_neighbours()[1], b.get_neighbours()[1]
                assert np.array_equal(ids, ref_ids)
                assert np.array_equal(a.get_state()["speed"], b.get_state()["speed"])
        for _ in range(2):  # and plain ticks after it
            a.step(1, neighbours=True)
            b.step(1, neighbours=True)
        ref = a.get_state()
        ref["count"] = a.get_neighbours(with_idx=False)[0]
        _same(ref, b.get_state(), b.get_neighbours(with_idx=False)[0], "after plain ticks")
        for buf in bufs.values():
            buf.free()


def test_direct_host_tick_refuses_a_bad_heading(msim):
    """The entity is named, the context keeps its state and serves the mended arrays."""
    road_map = msim.RoadMap.lattice(16, 2)
    n = 70_001
    kw = dict(rng="pcg32", dt=0.1, radius=2.0, cap=4)
    with msim.Simulation(road_map, n, **kw) as a, msim.Simulation(road_map, n, **kw) as b:
        a.init_entities(1, placement="fraction", speed=(1.0, 1.6))
        bufs, state = _pinned(msim, a.get_state(), n, True)
        for _ in range(3):
            a.tick_host(state, neighbours=True, out=state)
        before = a.get_state()
        for bad in (69_999, 12):
            state["heading"][bad] = road_map.num_roads
        with pytest.raises(msim.MsimError) as e:
            a.tick_host(state, neighbours=True, out=state)
        assert e.value.code == 2 and "entity 12 " in str(e.value)
        after = a.get_state()
        assert all(np.array_equal(before[k], after[k]) for k in before) and a.tick == 3
        for k in ("pos", "heading", "rng"):
            state[k][...] = before[k]
        for t in range(3):
            b.set_entities(state["pos"], state["heading"], state["rng"], state["speed"])
            b.step(1, neighbours=True)
            a.tick_host(state, neighbours=True, out=state)
            _same(state, b.get_state(), b.get_neighbours(with_idx=False)[0], f"at tick {t + 1}")
        for buf in bufs.values():
            buf.free()
