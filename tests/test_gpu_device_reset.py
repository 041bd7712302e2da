"""Contexts created after the device's CUDA context was reset (cudaDeviceReset by another
part of the program, all contexts of the library closed): they work as the first ones did.
In a process of its own, since a reset ends every other user of the CUDA context."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

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


def test_contexts_after_a_device_reset():
    got = subprocess.run([sys.executable, "-c", SCRIPT.format(root=str(ROOT))], capture_output=True, text=True,
                         timeout=300)
    assert got.returncode == 0 and got.stdout.strip() == "same", got.stdout + got.stderr
