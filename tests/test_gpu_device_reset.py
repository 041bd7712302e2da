"""Contexts created after the device's CUDA context was reset (cudaDeviceReset by another
part of the program, all contexts of the library closed): they work as the first ones did.
In a process of its own, since a reset ends every other user of the CUDA context."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

NOALLOC = """
import ctypes, importlib, sys
sys.path.insert(0, {root!r})
import numpy as np
msim = importlib.import_module("movement-sim_gb300")
fn = msim.lib().msim_query_neighbours_noalloc
vp, u32, f32 = ctypes.c_void_p, ctypes.c_uint32, ctypes.c_float
fn.restype, fn.argtypes = ctypes.c_int, [vp, u32, f32, f32, f32, u32, vp, vp, vp, vp]
cu, device, n, cap = ctypes.CDLL("libcuda.so.1"), ctypes.c_int(), 20_000, 200
pos = np.random.default_rng(1).uniform(0, 300, (n, 2)).astype(np.float32)
out = np.empty(n * (cap + 1), np.uint32)
def run():
    msim.set_device(0)
    a, b = ctypes.c_uint64(), ctypes.c_uint64()
    assert cu.cuMemAlloc_v2(ctypes.byref(a), ctypes.c_size_t(pos.nbytes)) == 0
    assert cu.cuMemAlloc_v2(ctypes.byref(b), ctypes.c_size_t(out.nbytes)) == 0
    assert cu.cuMemcpyHtoD_v2(a, vp(pos.ctypes.data), ctypes.c_size_t(pos.nbytes)) == 0
    for _ in range(2):
        assert fn(a.value, n, 300.0, 300.0, 2.0, cap, b.value, b.value + 4 * n, None, None) == 0
    assert cu.cuMemcpyDtoH_v2(vp(out.ctypes.data), b, ctypes.c_size_t(out.nbytes)) == 0
    assert cu.cuMemFree_v2(a) == 0 and cu.cuMemFree_v2(b) == 0
    assert out[:n].max() > 0
    return out.tobytes()
first = run()
assert cu.cuDeviceGet(ctypes.byref(device), 0) == 0
assert cu.cuDevicePrimaryCtxReset_v2(device) == 0
assert run() == first
print("same")
"""

SCRIPT = """
import ctypes, importlib, sys
sys.path.insert(0, {root!r})
import numpy as np
msim = importlib.import_module("movement-sim_gb300")
road_map = msim.RoadMap.lattice(16, 3)
def run():
    out = []
    with msim.Simulation(road_map, 5000, rng="pcg32", dt=0.1, radius=2.0, cap=8) as sim:
        sim.init_entities(4, placement="fraction", speed=(1.0, 1.6))
        sim.step(3, neighbours=True)
        out += [*sim.get_state().values(), *sim.get_neighbours(), np.uint64(sim.collision_pairs())]
        state = sim.get_state()
        for _ in range(2):
            state = sim.tick_host(state, neighbours=True) | {{"speed": state["speed"]}}
        out += list(state.values())
    with msim.Batch([road_map, road_map], [3000, 500]) as batch:
        batch.init_entities([1, 2])
        batch.step(5)
        out += [v for i in range(2) for v in batch.get_state(i).values()]
    return [np.asarray(v).tobytes() for v in out]
first = run()
cu, device = ctypes.CDLL("libcuda.so.1"), ctypes.c_int()
assert cu.cuDeviceGet(ctypes.byref(device), 0) == 0
for _ in range(2):
    assert cu.cuDevicePrimaryCtxReset_v2(device) == 0
    assert run() == first
print("same")
"""


@pytest.mark.parametrize("script", [SCRIPT, NOALLOC], ids=["contexts", "no_allocation_query"])
def test_after_a_device_reset(script):
    got = subprocess.run([sys.executable, "-c", script.format(root=str(ROOT))], capture_output=True, text=True,
                         timeout=300)
    assert got.returncode == 0 and got.stdout.strip() == "same", got.stdout + got.stderr
