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
