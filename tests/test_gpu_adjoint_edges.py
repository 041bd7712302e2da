"""Calibration at the sizes where its kernels divide the work: one entity, a warp's
share plus or minus one, fewer and more than one entity per lane of the chip, tick
counts around a schedule word, checkpoints that do not divide it, segments longer than
the run, one cell, odd and wide grids; against the FP64 adjoint.

Tolerances: the density is a sum of integer weights of 2^-31 (1e-5 relative, as the
main test).  The backward recomputes positions to a rounding per tick (at most K half
units of a coordinate, about 5e-4 m here, against steps of 0.1 m and more): one tick
in about two hundred cell crossings lands in the neighbouring cell, which changes that
entity's gradient by about one tick in `ticks`.  Averaged over a thousand entities
that stays below 1e-3; for a handful a single such tick is allowed, 1 / ticks at most
(5e-2)."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ticks,K,grid,rng", [
    (1, 1, 1, (1, 1), "pcg32"),
    (31, 32, 100, (64, 64), "pcg32"),
    (33, 33, 7, (5, 3), "xorshift128"),
    (1000, 31, 32, (7, 200), "pcg32"),
    (1217, 64, 33, (33, 31), "xorshift128"),
    (9729, 65, 64, (512, 16), "pcg32"),
    (40_001, 40, 13, (64, 96), "xorshift128"),
])
def test_edges_match_fp64_reference(msim, orc, n, ticks, K, grid, rng):
    torch = pytest.importorskip("torch")
    cal_mod = importlib.import_module("movement-sim_gb300.calibration")
    road_map = msim.RoadMap.lattice(16, 3)
    rs = np.random.default_rng(n)
    dt = 0.5
    with cal_mod.Calibration(road_map, n, ticks, dt=dt, rng=rng, checkpoint_interval=K, grid=grid, seed=9) as calib:
        st = calib.initial_state()
        speed = torch.from_numpy(rs.uniform(1.0, 1.6, n).astype(np.float32)).cuda()
        factor = torch.from_numpy(rs.uniform(0.7, 1.3, road_map.num_roads).astype(np.float32)).cuda()
        target = torch.from_numpy(rs.uniform(0, 2.0 * n / (grid[0] * grid[1]), grid[0] * grid[1]).astype(np.float32)).cuda()
        dens = torch.empty_like(target)
        out = []
        for mode in ("natural", "replay", "natural"):
            loss = calib.forward(speed, factor, target, dens, mode=mode)
            gs, gf = torch.empty_like(speed), torch.empty_like(factor)
            calib.backward(gs, gf)
            out.append((loss, dens.cpu().numpy(), gs.cpu().numpy(), gf.cpu().numpy()))
        gs64, gf64 = calib.gradients_f64()
    for other in out[1:]:  # a replay of the run's own events and a second run are the same run
        assert other[0] == out[0][0]
        for a, b in zip(out[0][1:], other[1:]):
            assert np.array_equal(a, b)
    loss, dens, gs, gf = out[0]
    assert np.array_equal(gs, gs64.astype(np.float32)) and np.array_equal(gf, gf64.astype(np.float32))
    rl, rd, rgs, rgf = orc.density_adjoint(road_map, st, speed.cpu().numpy(), factor.cpu().numpy(),
                                           1 if rng == "pcg32" else 0, dt, ticks, grid, target.cpu().numpy())
    assert abs(loss - rl) <= 1e-6 * abs(rl)
    np.testing.assert_allclose(dens, rd, rtol=1e-5, atol=1e-6 * max(rd.max(), 1e-30))
    tol = 1e-3 if n >= 1000 else 5e-2
    for g, r in ((gs64, rgs), (gf64, rgf)):
        assert np.linalg.norm(g - r) <= tol * np.linalg.norm(r) + 1e-12
