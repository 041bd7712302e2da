"""Performance cases of the per-tick path: what a user of the library has it do.

Each case is one pass through the public entry points (`Simulation`, `Batch`,
`Calibration` and the allocation-free neighbour query) at the sizes of the
repository's configurations and tests: `listed()` names twelve, `draw(rng)` gives
more of the same ranges, `prepare` / `run` build and run one, `work` counts the bytes
and operations a pass cannot do without, and `exact` restates the computed values in
64 bits with torch alone.

Road maps are jittered lattices (50 m spacing, +-10 m, nine of ten edges kept), made
here with numpy; entities come from the library's documented initializer (counter
draws from a seed), restated here for `exact`.
"""
from __future__ import annotations

import ctypes
import functools
import importlib
import math

import numpy as np
import torch

msim = importlib.import_module("movement-sim_gb300")

# ---- the cases -------------------------------------------------------------------


def _step(name, n, side, ticks, **more):
    case = {"kind": "step", "n": n, "side": side, "ticks": ticks, "nbr": True, "rng": "pcg32", "dt": 0.1, "smin": 1.0,
            "smax": 1.6, "radius": 2.0, "cap": 64, "ids": False, "factors": False, **more}
    return {"name": name, **case} if name else case


def listed():
    return [
        # The plain configuration: a small simulation advanced its whole run, no neighbours.
        _step("plain_10k", 10_000, 32, 1000, nbr=False),
        # The same without neighbours at a size that fills the chip, per-road speed factors set.
        _step("plain_1m", 1_000_000, 256, 200, nbr=False, factors=True),
        # A small interactive simulation: one neighbour tick a call, everything read back.
        _step("tick_3k", 3_001, 16, 1, ids=True),
        # The reference's own mode: a million entities, 1.4 m a tick, 10 m radius, xorshift128.
        _step("reference_1m", 1_000_000, 256, 10, rng="xorshift128", dt=1.0, smin=1.4, smax=1.4, radius=10.0),
        # The neighbour configuration, read back every 25 ticks.
        _step("neighbours_1m", 1_000_000, 256, 25),
        # The scale configuration, the headline workload, read back every 20 ticks.
        _step("scale_16m", 16_000_000, 1024, 20),
        # A crowded town: about a dozen neighbours within 10 m, the id lists read back.
        _step("crowd_200k", 200_003, 64, 5, radius=10.0, ids=True),
        # A program that owns the state on the host: one tick a call, in place.
        {"name": "host_1m", "kind": "host", "n": 1_000_000, "side": 256, "rng": "pcg32", "dt": 0.1, "smin": 1.0,
         "smax": 1.6, "radius": 2.0, "cap": 64},
        # An ensemble of uneven instances (side 16 to 256, 1,000 to 200,000 entities) for its 1,000 ticks.
        {"name": "ensemble_20", "kind": "ensemble", "count": 20, "sizes": 1, "side_lo": 16, "side_hi": 256,
         "n_lo": 1_000, "n_hi": 200_000, "ticks": 1000, "rng": "pcg32", "dt": 0.1},
        # One training step of the calibration configuration (loss and both gradients).
        {"name": "calibration_262k", "kind": "calibration", "n": 262_144, "side": 128, "ticks": 2000, "every": 100,
         "grid_w": 512, "grid_h": 512, "rng": "pcg32", "dt": 0.1, "direct": False},
        # A small calibration, density read too (the tests' size).
        {"name": "calibration_6k", "kind": "calibration", "n": 6_000, "side": 16, "ticks": 300, "every": 50,
         "grid_w": 64, "grid_h": 64, "rng": "pcg32", "dt": 0.1, "direct": True},
        # Neighbour sets of positions a caller holds on the device, no allocation.
        {"name": "positions_100k", "kind": "positions", "n": 100_003, "side": 80, "radius": 2.0, "cap": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(n, per_road):
    """Lattice side with about per_road entities on a road (1.8 roads to a node)."""
    return max(4, min(1024, int(round(math.sqrt(n / (1.8 * per_road))))))


def draw(rng):
    kind = rng.choice(["plain", "tick", "neighbours", "reference", "crowd", "host", "ensemble", "calibration",
                       "positions"])
    gen = rng.choice(["pcg32", "xorshift128"])
    per_road = math.exp(rng.uniform(math.log(4), math.log(12)))
    if kind == "plain":
        n = _log(rng, 1_000, 2_000_000)
        return _step(None, n, _side(n, per_road), _log(rng, 64, 1000), nbr=False, rng=gen, factors=rng.random() < 0.5)
    if kind == "tick":
        n = _log(rng, 1_000, 100_000)
        return _step(None, n, _side(n, per_road), 1, rng=gen, cap=rng.choice([0, 8, 16, 64]), ids=rng.random() < 0.5,
                     radius=rng.uniform(1.0, 4.0))
    if kind == "neighbours":
        n = _log(rng, 20_000, 8_000_000)
        return _step(None, n, _side(n, per_road), rng.randint(5, 20), rng=gen, cap=rng.choice([0, 16, 64]),
                     factors=rng.random() < 0.25, radius=rng.uniform(1.0, 3.0))
    if kind == "reference":
        n = _log(rng, 20_000, 1_000_000)
        return _step(None, n, _side(n, rng.uniform(5, 9)), rng.randint(2, 10), rng="xorshift128", dt=1.0, smin=1.4,
                     smax=1.4, radius=10.0)
    if kind == "crowd":
        n = _log(rng, 20_000, 200_000)
        return _step(None, n, _side(n, rng.uniform(12, 27)), rng.randint(1, 5), rng=gen, radius=rng.uniform(6.0, 10.0),
                     cap=rng.choice([16, 64]), ids=rng.random() < 0.5)
    if kind == "host":
        n = _log(rng, 20_000, 2_000_000)
        return {"kind": "host", "n": n, "side": _side(n, per_road), "rng": gen, "dt": 0.1, "smin": 1.0, "smax": 1.6,
                "radius": rng.uniform(1.0, 3.0), "cap": rng.choice([16, 64])}
    if kind == "ensemble":
        return {"kind": "ensemble", "count": rng.randint(3, 20), "sizes": rng.randrange(1 << 20), "side_lo": 16,
                "side_hi": 128, "n_lo": 1_000, "n_hi": _log(rng, 5_000, 200_000), "ticks": _log(rng, 100, 1000),
                "rng": gen, "dt": 0.1}
    if kind == "calibration":
        n = _log(rng, 2_000, 262_144)
        ticks = _log(rng, 100, 1500)
        return {"kind": "calibration", "n": n, "side": _side(n, per_road), "ticks": ticks,
                "every": rng.choice([25, 50, 64, 100]), "grid_w": _log(rng, 48, 512), "grid_h": _log(rng, 48, 512),
                "rng": gen, "dt": 0.1, "direct": rng.random() < 0.5}
    n = _log(rng, 1_000, 262_144)
    return {"kind": "positions", "n": n, "side": _side(n, per_road), "radius": rng.uniform(1.0, 4.0),
            "cap": rng.choice([0, 8, 16, 64])}


# ---- inputs ----------------------------------------------------------------------


@functools.lru_cache(maxsize=64)
def _lattice(side, seed):
    """A jittered lattice in the map layout.  A road end with three or more entries draws
    one of the entries 1 .. count after its first (one with two always takes entry 1),
    so a node's list is one entry to skip, then its roads, twice over where there are
    two: every road of a node is drawn equally often, and a population stays spread out
    however long it runs."""
    g = np.random.default_rng([side, seed])
    node = np.arange(side * side)
    a, b = node % side, node // side
    xy = (50.0 * np.stack([a, b], 1) + 20.0 * g.random((side * side, 2))).astype(np.float32)
    right, up = (g.random(side * side) < 0.9) & (a + 1 < side), (g.random(side * side) < 0.9) & (b + 1 < side)
    start = np.concatenate([node[right], node[up]])
    end = np.concatenate([node[right] + 1, node[up] + side])
    order = np.argsort(start, kind="stable")
    start, end = start[order], end[order]
    road = np.arange(start.size)
    at, conn = np.concatenate([start, end]), np.concatenate([road, road])
    two = np.bincount(at, minlength=side * side)[at] == 2
    at, conn = np.append(at, at[two]), np.append(conn, conn[two])
    order = np.argsort(at, kind="stable")  # by node
    at, conn = at[order], conn[order]
    count = np.bincount(at, minlength=side * side)
    first = np.concatenate([[0], np.cumsum(count)])[:-1]
    used = np.unique(at)
    conn = np.insert(conn, first[used], conn[first[used]]).astype(np.uint32)  # the entry to skip
    begins = first + np.cumsum(count > 0) - (count > 0)
    road_pos = np.concatenate([xy[start], xy[end]], 1)
    road_conn = np.stack([begins[start], count[start], begins[end], count[end]], 1).astype(np.uint32)
    width, height = xy[np.concatenate([start, end])].max(0)
    return msim.RoadMap(road_pos, road_conn, conn, float(width), float(height))


def _sizes(case):
    g = np.random.default_rng(case["sizes"])
    sides = g.integers(case["side_lo"], case["side_hi"] + 1, case["count"])
    n = np.floor(np.exp(g.uniform(math.log(case["n_lo"]), math.log(case["n_hi"]), case["count"])))
    return [(int(s), int(k)) for s, k in zip(sides, n)]


def _pinned(shape, dtype):
    """Page-locked array (kept alive by whoever holds a view of it)."""
    kind = {np.float32: torch.float32, np.uint32: torch.int32}[dtype]
    return torch.empty(shape, dtype=kind, pin_memory=True).numpy().view(dtype)


def _factors(roads, seed):
    return np.random.default_rng(seed + 17).uniform(0.7, 1.3, roads).astype(np.float32)


def _state_arrays(n):
    return {"pos": _pinned((n, 2), np.float32), "heading": _pinned((n,), np.uint32), "rng": _pinned((n, 4), np.uint32)}


def prepare(case, seed):
    if torch.cuda.is_available():
        torch.cuda.init()
    kind = case["kind"]
    if kind == "ensemble":
        sizes = _sizes(case)
        batch = msim.Batch([_lattice(s, k) for k, (s, _) in enumerate(sizes)], [n for _, n in sizes], rng=case["rng"],
                           dt=case["dt"])
        batch.init_entities([seed + k for k in range(len(sizes))])
        return {"case": case, "batch": batch}
    road_map = _lattice(case["side"], 0)
    n = case["n"]
    if kind == "step":
        sim = msim.Simulation(road_map, n, rng=case["rng"], dt=case["dt"], radius=case["radius"], cap=case["cap"])
        sim.init_entities(seed, placement="fraction", speed=(case["smin"], case["smax"]))
        if case["factors"]:
            sim.set_road_factors(_factors(road_map.num_roads, seed))
        out = _state_arrays(n)
        nbr = (_pinned((n,), np.uint32), _pinned((n, max(case["cap"], 1)), np.uint32) if case["ids"] else None)
        return {"case": case, "sim": sim, "out": out, "nbr": nbr}
    if kind == "host":
        sim = msim.Simulation(road_map, n, rng=case["rng"], dt=case["dt"], radius=case["radius"], cap=case["cap"])
        e = _entities(road_map, n, seed, case["rng"], case["smin"], case["smax"])
        state = {**_state_arrays(n), "speed": _pinned((n,), np.float32)}
        state["pos"][:] = e["pos"].cpu().numpy()
        state["heading"][:] = _heading(e["road"], e["to_end"]).cpu().numpy().astype(np.uint32)
        state["rng"][:] = e["rng"].cpu().numpy().astype(np.uint32)
        state["speed"][:] = e["speed"].cpu().numpy()
        out = {"pos": state["pos"], "heading": state["heading"], "rng": state["rng"], "count": _pinned((n,), np.uint32)}
        return {"case": case, "sim": sim, "state": state, "out": out}
    if kind == "calibration":
        calibration = importlib.import_module("movement-sim_gb300.calibration")
        calib = calibration.Calibration(road_map, n, case["ticks"], dt=case["dt"], rng=case["rng"],
                                        checkpoint_interval=case["every"], grid=(case["grid_w"], case["grid_h"]),
                                        seed=seed)
        speed, factor, target = _calibration_inputs(case, seed, road_map)
        return {"case": case, "calib": calib, "loss": calibration.density_loss, "speed": speed.requires_grad_(),
                "factor": factor.requires_grad_(), "target": target, "density": torch.empty_like(target),
                "grads": (torch.empty_like(speed), torch.empty_like(factor))}
    fn = msim.lib().msim_query_neighbours_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_void_p, ctypes.c_uint32, ctypes.c_float, ctypes.c_float, ctypes.c_float, ctypes.c_uint32,
                   ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    pos = _entities(road_map, n, seed, "pcg32", 1.0, 1.6)["pos"].contiguous()
    return {"case": case, "fn": fn, "world": (road_map.width, road_map.height), "pos": pos,
            "count": torch.empty(n, dtype=torch.int32, device=pos.device),
            "idx": torch.empty((n, max(case["cap"], 1)), dtype=torch.int32, device=pos.device)}


def _words(got):
    """Words as int32 views (torch has few operations on uint32)."""
    return {k: v.view(np.int32) if v.dtype == np.uint32 else v for k, v in got.items()}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        sim, out = state["sim"], state["out"]
        sim.step(case["ticks"], neighbours=case["nbr"])
        sim.get_state(out)
        got = dict(out)
        if case["nbr"]:
            ids = case["ids"] and case["cap"] > 0
            got["count"], idx = sim.get_neighbours(with_idx=ids, out=state["nbr"])
            if ids:
                got["ids"] = idx
        return _words(got)
    if kind == "host":
        return _words(state["sim"].tick_host(state["state"], neighbours=True, out=state["out"]))
    if kind == "ensemble":
        batch = state["batch"]
        batch.step(case["ticks"])
        got = []
        for k in range(case["count"]):
            s = batch.get_state(k)
            got.append(_words({"pos": s["pos"], "heading": s["heading"], "rng": s["rng"]}))
        return got
    if kind == "calibration":
        if case["direct"]:
            calib, (gs, gf) = state["calib"], state["grads"]
            loss = calib.forward(state["speed"].detach(), state["factor"].detach(), state["target"], state["density"])
            calib.backward(gs, gf)
            return {"loss": loss, "density": state["density"], "speed": gs, "factor": gf}
        loss = state["loss"](state["calib"], state["speed"], state["factor"], state["target"])
        gs, gf = torch.autograd.grad(loss, (state["speed"], state["factor"]))
        return {"loss": loss.detach(), "speed": gs, "factor": gf}
    pos, cap = state["pos"], case["cap"]
    rc = state["fn"](pos.data_ptr(), case["n"], *state["world"], case["radius"], cap, state["count"].data_ptr(),
                     state["idx"].data_ptr() if cap else None, None, torch.cuda.current_stream().cuda_stream)
    if rc:
        raise RuntimeError(msim.lib().msim_last_error().decode())
    return {"count": state["count"], "ids": state["idx"]} if cap else {"count": state["count"]}


# ---- work ------------------------------------------------------------------------

MOVE_FLOPS = 14  # two differences, the distance, two divisions, two scaled steps, the comparison
PAIR_FLOPS = 6   # difference, squares, sum, comparison


def work(case):
    """A move-only run keeps the state on the chip: read and written once.  A neighbour
    tick reads and writes every position and reads the positions again by place, for
    its counts; the state is larger than the chip holds beside the maps."""
    kind = case["kind"]
    if kind == "ensemble":
        n = sum(k for _, k in _sizes(case))
        return {"bytes": n * (32 + 28), "flops": MOVE_FLOPS * n * case["ticks"]}
    n = case["n"]
    if kind == "step" and not case["nbr"]:
        return {"bytes": n * (32 + 28), "flops": MOVE_FLOPS * n * case["ticks"]}
    if kind == "step":
        # entities within the radius: along the road, both ways
        near = max(1.0, 2.0 * case["radius"] * n / (1.8 * case["side"] ** 2 * 50.0))
        tick = 8 + 8 + 4 + 4 + 8 + 4 + 4 * min(near, case["cap"])
        back = 28 + 4 + (4 * case["cap"] if case["ids"] else 0)
        return {"bytes": n * (tick * case["ticks"] + back), "flops": (MOVE_FLOPS + PAIR_FLOPS * near) * n * case["ticks"]}
    if kind == "host":
        return {"bytes": n * (32 + 8 + 4), "flops": (MOVE_FLOPS + PAIR_FLOPS) * n}
    if kind == "calibration":
        # forward: move, splat position read; backward: recompute or read back, adjoint
        steps = n * case["ticks"]
        return {"bytes": 16.0 * steps + 12.0 * case["grid_w"] * case["grid_h"], "flops": 3.0 * MOVE_FLOPS * steps}
    return {"bytes": n * (8 + 4 + 4 * case["cap"]), "flops": PAIR_FLOPS * 2 * n}


# ---- the same values in 64 bits ----------------------------------------------------

_M64 = (1 << 64) - 1
_M32 = 0xFFFFFFFF


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _signed(v):
    v &= _M64
    return v - (1 << 64) if v >> 63 else v


def _shr(z, k):
    """Logical right shift of 64-bit words."""
    return (z >> k) & ((1 << (64 - k)) - 1)


def _mix(z):
    z = z + _signed(0x9E3779B97F4A7C15)
    z = (z ^ _shr(z, 30)) * _signed(0xBF58476D1CE4E5B9)
    z = (z ^ _shr(z, 27)) * _signed(0x94D049BB133111EB)
    return z ^ _shr(z, 31)


def _counter(seed, stream, i):
    first = _mix(torch.tensor([_signed(seed + 0x632BE59BD9B4E019 * stream)], dtype=torch.int64, device=i.device))
    return _mix(first + i)


def _unit(d):
    return _shr(d, 40).to(torch.float32) * 2.0 ** -24


def _pcg_next(state, inc):
    return state * 6364136223846793005 + inc


def _entities(road_map, n, seed, gen, smin, smax):
    """The initializer's entities (uniform fraction along a uniform road)."""
    i = torch.arange(n, dtype=torch.int64, device=_device())
    rp = torch.from_numpy(road_map.road_pos).to(i.device)
    road = _shr(_shr(_counter(seed, 1, i), 32) * road_map.num_roads, 32)
    at = rp[road]
    u = _unit(_counter(seed, 2, i))
    pos = torch.stack([at[:, 0] + u * (at[:, 2] - at[:, 0]), at[:, 1] + u * (at[:, 3] - at[:, 1])], 1)
    lo = torch.tensor(smin, dtype=torch.float32, device=i.device)
    hi = torch.tensor(smax, dtype=torch.float32, device=i.device)
    speed = lo + _unit(_counter(seed, 3, i)) * (hi - lo)
    a, b = _counter(seed, 4, i), _counter(seed, 5, i)
    if gen == "pcg32":
        inc = b * 2 + 1
        state = _pcg_next(_pcg_next(torch.zeros_like(a), inc) + a, inc)
        words = [state & _M32, _shr(state, 32), inc & _M32, _shr(inc, 32)]
    else:
        words = [a & _M32, _shr(a, 32), b & _M32, _shr(b, 32)]
        words[0] = torch.where((words[0] | words[1] | words[2] | words[3]) == 0, torch.ones_like(a), words[0])
    return {"pos": pos, "road": road, "to_end": torch.ones(n, dtype=torch.bool, device=i.device), "speed": speed,
            "rng": torch.stack(words, 1)}


def _heading(road, to_end):
    return road | (to_end.to(torch.int64) << 31)


def _next_random(rng, who, gen):
    """The next 32 random bits of the entities `who`; their states move on."""
    w = rng[who]
    if gen == "pcg32":
        old, inc = w[:, 0] | (w[:, 1] << 32), w[:, 2] | (w[:, 3] << 32)
        new = _pcg_next(old, inc)
        rng[who, 0], rng[who, 1] = new & _M32, _shr(new, 32)
        bits = _shr(_shr(old, 18) ^ old, 27) & _M32
        rot = _shr(old, 59)
        return ((bits >> rot) | (bits << (32 - rot))) & _M32
    t, s = w[:, 3], w[:, 0]
    t = t ^ ((t << 11) & _M32)
    t = t ^ (t >> 8)
    t = t ^ s ^ (s >> 19)
    rng[who] = torch.stack([t, s, w[:, 1], w[:, 2]], 1)
    return t


def _advance(road_map, e, ticks, dt, gen, dtype, factor=None, seen=None):
    """`ticks` move ticks of the entities e in `dtype`; seen(x, y, road, target, event)
    is told each tick's new position, the road and target before it and who arrived."""
    dev = e["pos"].device
    rp = torch.from_numpy(road_map.road_pos).to(dev).to(dtype)
    rc = torch.from_numpy(road_map.road_conn.astype(np.int64)).to(dev)
    conn = torch.from_numpy(np.append(road_map.connections, road_map.connections[-1:]).astype(np.int64)).to(dev)
    x, y = e["pos"][:, 0].to(dtype), e["pos"][:, 1].to(dtype)
    road, to_end, rng = e["road"].clone(), e["to_end"].clone(), e["rng"].clone()
    speed = e["speed"].to(dtype)
    dt = torch.tensor(dt, dtype=torch.float32, device=dev).to(dtype)
    fac = None if factor is None else factor.to(dtype)
    ends = torch.where(to_end[:, None], rp[road, 2:], rp[road, :2])
    tx, ty = ends[:, 0].clone(), ends[:, 1].clone()
    step = (speed if fac is None else speed * fac[road]) * dt
    for _ in range(ticks):
        dx, dy = tx - x, ty - y
        dist = torch.sqrt((dx * dx + dy * dy).double()).to(dtype)  # correctly rounded in either type
        go = dist > step
        x = torch.where(go, x + dx / dist * step, tx)
        y = torch.where(go, y + dy / dist * step, ty)
        if seen:
            seen(x, y, road, tx, ty, ~go)
        who = (~go).nonzero()[:, 0]
        if not who.numel():
            continue
        old, end = road[who], to_end[who]
        ix = torch.where(end, rc[old, 2], rc[old, 0])
        count = torch.where(end, rc[old, 3], rc[old, 1])
        off = torch.ones_like(ix)
        many = (count > 2).nonzero()[:, 0]
        if many.numel():  # the draw in binary32, as the shader does
            f = _next_random(rng, who[many], gen).to(torch.float32) * 2.0 ** -32
            off[many] = torch.ceil(1.0 + f * count[many].to(torch.float32)).to(torch.int64) - 1
        new = torch.where(count <= 1, old, conn[torch.clamp(ix + off, max=conn.numel() - 1)])
        starts = (rp[new, 0] == tx[who]) & (rp[new, 1] == ty[who])
        end = torch.where(count <= 1, ~end, starts)
        road, to_end = road.clone(), to_end.clone()
        road[who], to_end[who] = new, end
        aim = torch.where(end[:, None], rp[new, 2:], rp[new, :2])
        tx, ty = tx.clone(), ty.clone()
        tx[who], ty[who] = aim[:, 0], aim[:, 1]
        if fac is not None:
            step[who] = speed[who] * fac[new] * dt
    return torch.stack([x, y], 1)


def _corners(case, road_map, x, y):
    """Cell-centred bilinear weights: per corner (inside, flat cell, column and row weight)."""
    gw, gh = case["grid_w"], case["grid_h"]
    u, v = x.double() * (gw / road_map.width) - 0.5, y.double() * (gh / road_map.height) - 0.5
    i, j = torch.floor(u), torch.floor(v)
    fx, fy = u - i, v - j
    for di, wx in ((0, 1.0 - fx), (1, fx)):
        for dj, wy in ((0, 1.0 - fy), (1, fy)):
            ci, cj = i.long() + di, j.long() + dj
            inside = (ci >= 0) & (cj >= 0) & (ci < gw) & (cj < gh)
            yield di, dj, inside, torch.where(inside, cj * gw + ci, torch.zeros_like(ci)), wx, wy


def _calibration_inputs(case, seed, road_map):
    """Speeds, road factors and a target density: another population's positions, smoothed."""
    dev = _device()
    speed = _entities(road_map, case["n"], seed + 1, case["rng"], 1.0, 1.6)["speed"].contiguous()
    factor = torch.from_numpy(_factors(road_map.num_roads, seed)).to(dev)
    other = _entities(road_map, case["n"], seed + 2, case["rng"], 1.0, 1.6)["pos"]
    ci = (other[:, 0] * (case["grid_w"] / road_map.width)).long().clamp(0, case["grid_w"] - 1)
    cj = (other[:, 1] * (case["grid_h"] / road_map.height)).long().clamp(0, case["grid_h"] - 1)
    target = torch.bincount(cj * case["grid_w"] + ci, minlength=case["grid_w"] * case["grid_h"]).float()
    target = target.view(case["grid_h"], case["grid_w"])
    for axis in (0, 1):
        target = 0.5 * target + 0.25 * (torch.roll(target, 1, axis) + torch.roll(target, -1, axis))
    return speed, factor, target.reshape(-1).contiguous()


def _exact_calibration(case, seed):
    """Density, loss and adjoint in 64 bits about the binary32 trajectory: positions and
    road-end events are defined in binary32, in source order."""
    road_map = _lattice(case["side"], 0)
    e = _entities(road_map, case["n"], seed, case["rng"], 1.0, 1.6)
    speed, factor, target = _calibration_inputs(case, seed, road_map)
    e["speed"] = speed
    cells, ticks = case["grid_w"] * case["grid_h"], case["ticks"]
    density = torch.zeros(cells, dtype=torch.float64, device=speed.device)
    past = [(e["pos"][:, 0], e["pos"][:, 1], None, None, None, None)]

    def seen(x, y, road, tx, ty, event):
        for _, _, inside, cell, wx, wy in _corners(case, road_map, x, y):
            density.index_add_(0, cell, torch.where(inside, wx * wy, torch.zeros_like(wx)))
        past.append((x, y, road.int(), tx, ty, event))

    _advance(road_map, e, ticks, case["dt"], case["rng"], torch.float32, factor, seen)
    density /= ticks
    off = density - target.double()
    lam = 2.0 / cells * off
    dt = float(np.float32(case["dt"]))
    s, f = speed.double(), factor.double()
    ax, ay = torch.zeros_like(s), torch.zeros_like(s)
    gs, gf = torch.zeros_like(s), torch.zeros_like(f)
    sx, sy = case["grid_w"] / road_map.width / ticks, case["grid_h"] / road_map.height / ticks
    for t in range(ticks, 0, -1):
        x, y, road, tx, ty, event = past.pop()
        for di, dj, inside, cell, wx, wy in _corners(case, road_map, x, y):
            here = torch.where(inside, lam[cell], torch.zeros_like(s))
            ax += here * wy * (sx if di else -sx)
            ay += here * wx * (sy if dj else -sy)
        dx, dy = tx.double() - past[-1][0].double(), ty.double() - past[-1][1].double()
        dist = torch.sqrt(dx * dx + dy * dy)
        go = ~event & (dist > 0)
        inv = torch.where(go, 1.0 / dist, torch.zeros_like(dist))
        nx, ny = dx * inv, dy * inv
        road = road.long()
        g = nx * ax + ny * ay
        gs += g * f[road] * dt
        gf.index_add_(0, road, g * s * dt)
        k = s * f[road] * dt * inv
        ax, ay = ax - k * (ax - nx * g), ay - k * (ay - ny * g)
        ax[event] = 0.0
        ay[event] = 0.0
    loss = float((off * off).mean())
    if case["direct"]:
        return {"loss": loss, "density": density, "speed": gs, "factor": gf}
    return {"loss": loss, "speed": gs, "factor": gf}


def _moved(case, seed, side, map_seed, n, smin, smax, ticks):
    road_map = _lattice(side, map_seed)
    e = _entities(road_map, n, seed, case["rng"], smin, smax)
    factor = torch.from_numpy(_factors(road_map.num_roads, seed)).to(_device()) if case.get("factors") else None
    return _advance(road_map, e, ticks, case["dt"], case["rng"], torch.float64, factor)


def exact(case, seed):
    kind = case["kind"]
    if kind == "positions":
        return None  # whole numbers only
    if kind == "calibration":
        return _exact_calibration(case, seed)
    if kind == "ensemble":
        return [{"pos": _moved(case, seed + k, s, k, n, 1.0, 1.6, case["ticks"]), "heading": None, "rng": None}
                for k, (s, n) in enumerate(_sizes(case))]
    pos = _moved(case, seed, case["side"], 0, case["n"], case["smin"], case["smax"], case.get("ticks", 1))
    got = {"pos": pos, "heading": None, "rng": None}
    if case.get("nbr", True):
        got["count"] = None
        if case.get("ids") and case["cap"] > 0:
            got["ids"] = None
    return got
