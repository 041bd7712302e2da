"""The move step's root and quotients (msim_device.cuh root_reciprocal, quotient) against
the correctly rounded intrinsics: every squared distance of their range, random quotients
and the quotients nearest to a middle between two floats (tests/cpp/exact_root.cu).
And the ticks that leave their range (road ends at a coordinate of zero, huge and tiny
coordinates, non-finite positions) bit for bit against the oracle."""
import importlib.util
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent


def _recipe():
    spec = importlib.util.spec_from_file_location("msim_build_lib",
                                                  ROOT / "movement-sim_gb300" / "build_lib.py")
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_root_and_quotients_are_correctly_rounded(tmp_path):
    recipe = _recipe()
    exe = tmp_path / "exact_root"
    flags = [f for f in recipe.NVCC_FLAGS if f not in ("-Xcompiler", "-fPIC", "-Wall")]
    subprocess.run([recipe._nvcc(), *flags, str(ROOT / "tests" / "cpp" / "exact_root.cu"), "-o", str(exe)],
                   check=True, capture_output=True, timeout=300)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout.split()
    counts = [int(out[i]) for i in (1, 3, 5, 7, 9)]
    assert counts[:4] == [0, 0, 0, 0], out
    assert counts[4] > 10_000_000, out  # that many nearest-to-middle operands were tried


@pytest.mark.parametrize("scale", [1.0, 1e-12, 1e-25, 1e13, 1e25])
@pytest.mark.parametrize("ticks", [1, 130])
def test_ticks_outside_the_fast_range(msim, orc, scale, ticks):
    """A square of roads with corners at zero, scaled out of the fast path's range both
    ways; positions on, beside and far off their roads, infinite and NaN."""
    c = np.float32(100.0 * scale)
    corners = np.array([[0, 0], [c, 0], [c, c], [0, c]], np.float32)
    pos = np.concatenate([corners, np.roll(corners, -1, 0)], 1)
    conn = np.tile(np.array([0, 4, 0, 4], np.uint32), (4, 1))
    road_map = msim.RoadMap(pos, conn, np.array([0, 1, 2, 3, 0, 1], np.uint32), float(c), float(c))
    n = 4099
    rs = np.random.default_rng(3)
    p = (rs.uniform(0, 1, (n, 2)) * c).astype(np.float32)
    p[::7, 0] = 0.0
    p[::11, 1] = c
    p[5::97] *= np.float32(1e-30)
    p[6::97] = np.inf
    p[7::97, 0] = np.nan
    head = (rs.integers(0, 4, n).astype(np.uint32) | (rs.integers(0, 2, n).astype(np.uint32) << 31)).astype(np.uint32)
    rng = rs.integers(1, 2**32, (n, 4), dtype=np.uint64).astype(np.uint32)
    speed = (rs.uniform(0.5, 3.0, n) * scale).astype(np.float32)
    with msim.Simulation(road_map, n, rng="xorshift128", dt=1.0) as sim:
        sim.set_entities(p, head, rng, speed)
        sim.step(ticks)
        st = sim.get_state()
    orc.step(road_map.road_pos, road_map.road_conn, road_map.connections, p, head, rng, speed, 0, 1.0, ticks)
    nan = np.isnan(p)
    assert np.array_equal(np.isnan(st["pos"]), nan)
    assert np.array_equal(st["pos"].view(np.uint32)[~nan], p.view(np.uint32)[~nan])
    assert np.array_equal(st["heading"], head) and np.array_equal(st["rng"], rng)
