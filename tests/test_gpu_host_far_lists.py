"""Host ticks with id lists, some after the host moved entities further than the radius:
lists below and above the size from which the host asks before it downloads them, arrays
page-locked and in place, page-locked apart, and pageable.  Compared bit for bit with the
same ticks through the separate calls (whole numbers and the same binary32 operations)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cap", [(1, 4), (20_001, 8), (70_001, 8), (70_001, 33)])
@pytest.mark.parametrize("arrays", ["in_place", "page_locked", "pageable"])
def test_far_moved_host_ticks_with_lists(msim, n, cap, arrays):
    road_map = msim.RoadMap.lattice(40, 3)
    kw = dict(rng="pcg32", dt=0.1, radius=2.0, cap=cap)
    with msim.Simulation(road_map, n, **kw) as a, msim.Simulation(road_map, n, **kw) as b:
        a.init_entities(4, placement="fraction", speed=(1.0, 1.6))
        st, keep = a.get_state(), []

        def array(shape, dtype):
            if arrays == "pageable":
                return np.empty(shape, dtype)
            keep.append(msim.PinnedBuffer(shape, dtype))
            return keep[-1].array

        state = {k: array(v.shape, v.dtype) for k, v in st.items()}
        for k in st:
            state[k][...] = st[k]
        out = {k: state[k] if arrays == "in_place" else array(st[k].shape, st[k].dtype)
               for k in ("pos", "heading", "rng")}
        out |= {"count": array(n, np.uint32), "idx": array((n, cap), np.uint32)}
        for t in range(7):
            if t in (2, 4, 5):
                state["pos"][t::9] += np.float32(3.0 if t < 5 else np.inf)
            b.set_entities(state["pos"], state["heading"], state["rng"], state["speed"])
            b.step(1, neighbours=True)
            a.tick_host(state, neighbours=True, out=out)
            ref = b.get_state() | dict(zip(("count", "idx"), b.get_neighbours()))
            for k in out:
                assert np.array_equal(out[k].view(np.uint32), ref[k].view(np.uint32)), f"{k} at tick {t + 1}"
            assert a.collision_pairs() == b.collision_pairs()
            for k in ("pos", "heading", "rng"):
                state[k][...] = out[k]
        del state, out
        for buf in keep:
            buf.free()
