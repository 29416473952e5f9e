"""Performance cases: what programs built on this package have it do.

Every case is one call sequence of a user's program through the public entry
points (`sim`, `step`, `ensemble`, `serve`, `calib`), on inputs made from a
seed. Eight kinds of use ("path"):

* step      one `Simulation.step()`: a program that owns its own time loop
* run       `Simulation.run_steps(n)`, optionally with gauges
* until     `Simulation.run_until(t + span)`: a coupling interval
* solve     host arrays in, `Simulation`, n steps, host arrays out
* free      one step of the free functions on CUDA tensors (CFL dt, stage(s),
            friction, rain, point sources)
* ensemble  n batch steps of uneven scenarios, and their states
* serve     a burst of requests admitted, advanced and collected
* tangent / gradient
            the Dual tangent (one or several lanes) and the adjoint of a
            gauge misfit

and five regimes of the flow:

* valley    terrain with hills, open sides, rain and an inflow hydrograph:
            a thin sheet on the slopes and deep water along the thalweg
* wet       deep water over a smooth bed, walls
* dam       circular dam break, walls
* dry       a wet channel in a dry V-shaped valley (about 6% wet), walls
* urban     blocks standing out of a gentle slope, rain and a point inflow
* river     a sloping channel with Discharge upstream and Depth downstream
"""
from __future__ import annotations

import math

import numpy as np
import torch

F64 = torch.float64
G, H_DRY, H_VEL, DRY_TOL = 9.81, 1.0e-6, 1.0e-5, 1.0e-12
RAIN = 50.0e-3 / 3600.0
N, S, W, E = 0, 1, 2, 3
OPEN, WALL, DISCHARGE, DEPTH = 0, 1, 2, 3


def listed():
    return [
        # A program with its own time loop (adaptive output, coupling to
        # another model) on a small pond: the latency of one step.
        {"name": "step_48x64", "path": "step", "regime": "wet", "rows": 48, "cols": 64},
        # The circular dam break at its usual size, advanced by a short
        # interval between outputs (about 25 steps).
        {"name": "until_dam_256", "path": "until", "regime": "dam", "rows": 256, "cols": 256,
         "span": 0.4},
        # An urban rain event at 2 m on an odd-sized DEM with control points:
        # the UK EA 8A deck's shape, 50 steps of it.
        {"name": "run_urban_199x481", "path": "run", "regime": "urban", "rows": 199, "cols": 481,
         "steps": 50, "gauges": 9},
        # A river reach driven by its boundary conditions, ragged in both
        # directions.
        {"name": "run_river_731x1003", "path": "run", "regime": "river", "rows": 731,
         "cols": 1003, "steps": 16, "gauges": 0},
        # The mostly dry regime of the reference's step benchmark, larger.
        {"name": "run_dry_2048", "path": "run", "regime": "dry", "rows": 2048, "cols": 2048,
         "steps": 8, "gauges": 0},
        # The headline workload: the valley flood at 4096 x 4096.
        {"name": "run_valley_4096", "path": "run", "regime": "valley", "rows": 4096, "cols": 4096,
         "steps": 3, "gauges": 0},
        # A whole solve from host arrays to host arrays: upload, graph
        # capture, steps, read back.
        {"name": "solve_valley_1024", "path": "solve", "regime": "valley", "rows": 1024,
         "cols": 1024, "steps": 16},
        # The crate's free functions on resident tensors, as a caller that
        # keeps its own state composes them.
        {"name": "free_ssprk2_700x500", "path": "free", "regime": "valley", "rows": 700,
         "cols": 500, "integrator": "ssprk2"},
        # An uneven ensemble (sides log-uniform) over one output interval.
        {"name": "ensemble_16", "path": "ensemble", "regime": "valley", "count": 16, "lo": 64,
         "hi": 640, "steps": 72},
        # A burst of requests served to their horizons.
        {"name": "serve_8", "path": "serve", "regime": "valley", "count": 8, "lo": 64, "hi": 512,
         "span": 12.0},
        # Vector-mode tangent on a small calibration grid (8 zones).
        {"name": "tangent_64_lanes8", "path": "tangent", "regime": "river", "rows": 64,
         "cols": 64, "steps": 40, "lanes": 8},
        # The Manning-field gradient of a gauge misfit at 512 x 512.
        {"name": "gradient_512", "path": "gradient", "regime": "river", "rows": 512, "cols": 512,
         "steps": 48, "lanes": 0},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    path = rng.choice(["step", "until", "run", "run", "run", "solve", "free", "ensemble", "serve",
                       "tangent", "gradient"])
    regime = rng.choice(["valley", "valley", "wet", "dry", "urban", "river"])
    if path == "step":
        return {"path": path, "regime": regime, "rows": size(16, 512), "cols": size(16, 512)}
    if path == "until":
        return {"path": path, "regime": "dam", "rows": size(96, 700), "cols": size(96, 700),
                "span": round(rng.uniform(0.1, 0.6), 3)}
    if path == "run":
        rows, cols = size(40, 2600), size(40, 2600)
        most = max(1, min(64, int(3.0e7 / (rows * cols))))
        return {"path": path, "regime": regime, "rows": rows, "cols": cols,
                "steps": rng.randint(1, most), "gauges": rng.choice([0, 0, 7])}
    if path == "solve":
        return {"path": path, "regime": regime, "rows": size(64, 1500), "cols": size(64, 1500),
                "steps": rng.randint(4, 14)}
    if path == "free":
        return {"path": path, "regime": regime, "rows": size(32, 2000), "cols": size(32, 2000),
                "integrator": rng.choice(["ssprk2", "euler"])}
    if path == "ensemble":
        return {"path": path, "regime": regime, "count": rng.randint(5, 18), "lo": size(32, 96),
                "hi": size(128, 700), "steps": rng.randint(8, 72)}
    if path == "serve":
        return {"path": path, "regime": regime, "count": rng.randint(4, 12), "lo": size(32, 96),
                "hi": size(128, 512), "span": round(rng.uniform(4.0, 12.0), 2)}
    rows, cols = size(40, 500), size(40, 500)
    return {"path": path, "regime": "river", "rows": rows, "cols": cols,
            "steps": rng.randint(16, 48),
            "lanes": rng.choice([1, 2, 5]) if path == "tangent" else 0}


# ------------------------------------------------------------------ inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Rng:
    """Seeded numbers on the host (a few per case)."""

    def __init__(self, seed):
        self.g = np.random.default_rng(seed)

    def u(self, lo, hi, n=None):
        v = self.g.uniform(lo, hi, n)
        return float(v) if n is None else [float(x) for x in v]


def _waves(rng, x, y, lx, ly, count=5):
    """A smooth random field of order 1."""
    f = torch.zeros((y.numel(), x.numel()), dtype=F64, device=x.device)
    for _ in range(count):
        kx, ky = rng.u(-6, 6) * math.pi / lx, rng.u(-6, 6) * math.pi / ly
        p = rng.u(0, 2 * math.pi)
        f += torch.cos(kx * x + p)[None, :] * torch.cos(ky * y + rng.u(0, 6.0))[:, None]
    return f / math.sqrt(count)


def _flow(regime, rows, cols, seed, smooth_n=False):
    """Mesh, state, boundaries and forcings of one solve, as tensors."""
    rng, dev = _Rng(seed), _device()
    dx = {"wet": 1.0, "dam": 1.0, "dry": 1.0, "urban": 2.0}.get(regime, 5.0)
    x = (torch.arange(cols, dtype=F64, device=dev) + 0.5) * dx
    y = (torch.arange(rows, dtype=F64, device=dev) + 0.5) * dx
    lx, ly = cols * dx, rows * dx
    wave = _waves(rng, x, y, lx, ly)
    f = {"rows": rows, "cols": cols, "dx": dx, "dy": dx, "cfl": 0.5, "rain": None, "src": [],
         "bcs": ((WALL, 0.0),) * 4}
    zero = torch.zeros((rows, cols), dtype=F64, device=dev)
    if regime in ("valley", "river"):
        side = 0.05 if regime == "valley" else 0.004
        bed = (0.005 * (ly - y))[:, None] + (side * (x - lx / 2).abs())[None, :]
        if regime == "valley":
            for _ in range(24):
                a, s = rng.u(1, 20), rng.u(20, 200)
                cx, cy = rng.u(0, lx), rng.u(0, ly)
                bed = bed + a * (torch.exp(-((y - cy) ** 2) / (2 * s * s))[:, None]
                                 * torch.exp(-((x - cx) ** 2) / (2 * s * s))[None, :])
            # a few millimetres of rain on the slopes, water up to 1.5 m deep
            # within 8% of the width of the thalweg
            film = 2.0e-3 + 1.0e-3 * wave.abs()
            deep = 1.5 * (1 - ((x - lx / 2).abs() / (0.04 * lx)) ** 2).clamp(min=0.0)
            h = film + deep[None, :] * (1.0 + 0.1 * wave)
            f["bcs"] = ((OPEN, 0.0),) * 4
            f["rain"] = ([0.0, 1800.0], [RAIN, 0.8 * RAIN])
            peak = 500.0 * rng.u(0.5, 2.0)
            f["src"] = [(0, cols // 2, [0.0, 1800.0, 3600.0], [0.1 * peak, peak, 0.1 * peak])]
        else:
            bed = bed + 0.1 * wave
            h = 1.5 + 0.2 * wave - (bed - (0.005 * (ly - y))[:, None]).clamp(max=1.0)
            h = h.clamp(min=0.2)
            q = rng.u(1.0, 2.0)
            f["bcs"] = ((DISCHARGE, q), (DEPTH, 1.5), (WALL, 0.0), (WALL, 0.0))
        hu, hv = 0.02 * wave * h, (0.5 + 0.1 * wave) * h
    elif regime in ("wet", "dam"):
        bed = 0.05 * wave if regime == "wet" else zero.clone()
        if regime == "wet":
            h = 1.0 + 0.2 * (y / ly)[:, None] + 0.1 * (x / lx)[None, :] + 0.05 * wave
        else:
            r = torch.sqrt((x - lx / 2)[None, :] ** 2 + (y - ly / 2)[:, None] ** 2)
            h = torch.where(r < 0.2 * min(lx, ly), 10.0 + 0.2 * wave, 1.0 + 0.02 * wave)
        hu, hv = 0.1 * h, 0.05 * h * (1 + 0.2 * wave)
    elif regime == "dry":
        bed = (0.05 * (x - lx / 2).abs())[None, :] + zero
        level = 0.05 * lx / 32
        h = (level * (1 + 0.02 * wave) - bed).clamp(min=0.0)
        hu, hv = zero.clone(), 0.1 * h
        f["cfl"] = 0.4
    elif regime == "urban":
        bed = (0.01 * (ly - y))[:, None] + (0.004 * (x - lx / 2).abs())[None, :] + 0.02 * wave
        for _ in range(max(4, rows * cols // 1200)):
            i, j = int(rng.u(0, rows)), int(rng.u(0, cols))
            hh, ww = int(rng.u(3, 14)), int(rng.u(3, 14))
            bed[i:i + hh, j:j + ww] = bed[i:i + hh, j:j + ww].amax() + 6.0
        h = 5.0e-3 + 2.0e-3 * wave.abs()
        hu, hv = zero.clone(), 0.05 * h
        f["cfl"] = 0.7
        f["rain"] = ([0.0, 60.0, 180.0], [8 * RAIN, 8 * RAIN, 2 * RAIN])
        f["src"] = [(rows // 3, cols // 2, [0.0, 600.0, 3600.0], [2.0, rng.u(4, 8), 1.0]),
                    (rows // 2, cols // 3, [0.0], [rng.u(0.5, 1.5)])]
    else:
        raise ValueError(regime)
    if smooth_n:
        n = torch.exp(math.log(0.04) + 0.3 * _waves(rng, x, y, lx, ly))
    else:  # four land-cover patches
        best = None
        n = zero
        for c in (0.025, 0.035, 0.05, 0.08):
            d = (y - rng.u(0, ly))[:, None] ** 2 + (x - rng.u(0, lx))[None, :] ** 2
            n = torch.full_like(zero, c) if best is None else torch.where(d < best, c, n)
            best = d if best is None else torch.minimum(best, d)
    f.update(z=bed.contiguous(), n=n.contiguous(), h=h.contiguous(), hu=hu.contiguous(),
             hv=hv.contiguous())
    return f


def _flows(case, seed):
    """The scenarios of an ensemble or a burst of requests (square, uneven)."""
    rng = _Rng(seed)
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    out = []
    for k in range(case["count"]):
        # the largest is always there, so that a case has one cost
        side = case["hi"] if k == 0 else int(round(math.exp(
            lo + (hi - lo) * ((k * 0.61803398875 + 0.1) % 1.0))))
        f = _flow(case["regime"], side, side, seed * 1009 + k)
        f["t_end"] = case.get("span", 1.0e9)
        if "span" in case:
            f["t_end"] *= rng.u(0.7, 1.0)
        out.append(f)
    return out


def _scenario(f):
    from hydroflux_b200.workloads import Scenario
    a = {k: f[k].cpu().numpy() for k in ("z", "n", "h", "hu", "hv")}
    arr = np.asarray
    return Scenario("case", a["z"], a["n"], f["dx"], f["dy"], a["h"], a["hu"], a["hv"],
                    bcs=f["bcs"], cfl=f["cfl"], t_end=f.get("t_end", 1.0e9),
                    rain=None if f["rain"] is None else tuple(arr(v) for v in f["rain"]),
                    sources=[(r, c, arr(t), arr(q)) for r, c, t, q in f["src"]])


def _bcs(f):
    from hydroflux_b200 import sim
    return sim.Boundaries2D(*[sim.Boundary(k, v) for k, v in f["bcs"]])


def _simulation(host, f):
    """A Simulation with the case's forcings, from host arrays."""
    from hydroflux_b200 import sim
    cfg = sim.SimulationConfig(cfl=f["cfl"], boundaries=_bcs(f))
    s = sim.Simulation(sim.Mesh2D(host["z"], f["dx"], f["dy"], host["n"]),
                       (host["h"], host["hu"], host["hv"]), cfg)
    if f["rain"] is not None:
        s.set_rain(list(zip(*f["rain"])))
    if f["src"]:
        s.set_point_sources([sim.PointSource(r, c, list(zip(t, q))) for r, c, t, q in f["src"]])
    return s


def _gauge_cells(case):
    k = case.get("gauges", 0)
    r, c = case["rows"], case["cols"]
    return [((2 * i + 1) * r // (2 * k), (i * 37 + c // 3) % c) for i in range(k)]


def _misfit(case, seed):
    """The calibration problem of the tangent and gradient cases."""
    f = _flow(case["regime"], case["rows"], case["cols"], seed, smooth_n=True)
    rng = np.random.default_rng(seed + 7)
    g = np.unique(rng.integers(0, case["rows"] * case["cols"], 16)).astype(np.int64)
    obs = rng.uniform(0.8, 1.6, (case["steps"], g.size))
    lanes = max(case["lanes"], 1)
    zones = torch.zeros((lanes, case["rows"], case["cols"]), dtype=F64, device=f["z"].device)
    edges = [case["cols"] * k // lanes for k in range(lanes + 1)]
    for k in range(lanes):  # zonal Manning parameters in vertical stripes
        zones[k, :, edges[k]:edges[k + 1]] = 0.04
    return f, g, obs, zones


def prepare(case, seed):
    path = case["path"]
    st = {"case": case}
    if path in ("ensemble", "serve"):
        scns = [_scenario(f) for f in _flows(case, seed)]
        st["count"] = len(scns)
        if path == "ensemble":
            from hydroflux_b200.ensemble import Ensemble
            st["ens"] = Ensemble(scns)
        else:
            from hydroflux_b200.serve import Server
            st["srv"], st["scns"] = Server(2 << 30, max_slots=64), scns
        return st
    if path in ("tangent", "gradient"):
        from hydroflux_b200.calib import Calibration
        f, g, obs, zones = _misfit(case, seed)
        st["cal"] = Calibration(_scenario(f), case["steps"], g, checkpoint_every=16)
        st["cal"].set_observations(obs)
        st["n"] = f["n"].cpu().numpy()
        st["dn"] = zones.cpu().numpy()
        return st
    f = _flow(case["regime"], case["rows"], case["cols"], seed)
    st["f"] = f
    if path == "free":
        from hydroflux_b200 import step
        st["mesh"] = step.DeviceMesh(f["z"], f["dx"], f["dy"], f["n"])
        st["ws"] = step.StepWorkspace2D.for_mesh(st["mesh"])
        st["bcs"] = _bcs(f)
        st["u"] = (f["h"], f["hu"], f["hv"])
        return st
    host = {k: f.pop(k).cpu().numpy() for k in ("z", "n", "h", "hu", "hv")}
    if path == "solve":
        st["host"] = host
        return st
    st["sim"] = _simulation(host, f)
    if case.get("gauges", 0):
        st["sim"].set_gauges(_gauge_cells(case), capacity=1 << 16)
    st["views"] = st["sim"].device_state()[:3]
    return st


# --------------------------------------------------------------------- run
def run(st):
    case = st["case"]
    path = case["path"]
    if path == "step":
        dt = st["sim"].step()
        return {"dt": dt, "u": st["views"]}
    if path == "run":
        st["sim"].run_steps(case["steps"])
        out = {"t": st["sim"].time(), "u": st["views"]}
        if case["gauges"]:
            out["peak"], out["last"] = st["sim"].gauge_peaks()
        return out
    if path == "until":
        st["sim"].run_until(st["sim"].time() + case["span"])
        return {"t": st["sim"].time(), "steps": st["sim"].steps(), "u": st["views"]}
    if path == "solve":
        with _simulation(st["host"], st["f"]) as s:
            s.run_steps(case["steps"])
            return {"t": s.time(), "u": s.states()}
    if path == "free":
        from hydroflux_b200 import step
        f, m, ws = st["f"], st["mesh"], st["ws"]
        h, hu, hv = st["u"]
        dt = min(step.cfl_time_step_with_bcs(h, hu, hv, m, st["bcs"], f["cfl"], ws), 60.0)
        one = step.ssprk2_step if case["integrator"] == "ssprk2" else step.forward_euler_step
        one(h, hu, hv, m, st["bcs"], dt, ws)
        step.manning_friction_step(h, hu, hv, m, dt, H_DRY)
        if f["rain"] is not None:
            step.apply_rain(h, hu, hv, f["rain"][1][0], dt)
        if f["src"]:
            step.apply_point_sources(h, hu, hv, [(r, c, q[0]) for r, c, _, q in f["src"]], dt,
                                     f["dx"], f["dy"])
        return {"dt": dt, "u": st["u"]}
    if path == "ensemble":
        e = st["ens"]
        left = e.run(case["steps"])
        return {"left": left, "t": [e.info(k)["t"] for k in range(st["count"])],
                "u": [e.states(k)[0] if k else e.states(k) for k in range(st["count"])]}
    if path == "serve":
        srv = st["srv"]
        slots = [srv.try_admit(s) for s in st["scns"]]
        got, waiting = {}, set(slots)
        while waiting:
            srv.advance(8)
            for slot in srv.finished():
                got[slot] = srv.collect(slot)
                waiting.discard(slot)
        return {"steps": [got[s]["steps"] for s in slots], "u": [got[s]["state"] for s in slots]}
    if path == "tangent":
        if case["lanes"] == 1:
            J, dJ = st["cal"].tangent(st["n"], st["dn"][0])
            return {"J": J, "dJ": dJ, "u": st["cal"].final_state()}
        J, dJ = st["cal"].tangent_lanes(st["n"], st["dn"])
        return {"J": J, "dJ": dJ, "lane0": st["cal"].lane_state(0)}
    J, g, g0 = st["cal"].gradient(st["n"], initial_state=True)
    return {"J": J, "gn": g, "g0": g0}


# -------------------------------------------------------------------- work
#: FP64 operations (+ - * / sqrt max, each one) of a cell: a forward-Euler
#: stage without halo work (primitives 3, slopes 24, two faces 170, alpha 11,
#: update and bed source 70) and the epilogue of a step (SSP-RK2 combination,
#: friction with its power, rain, CFL).
STAGE_OPS, EPILOGUE_OPS = 278, 70


def work(case):
    """A step reads h, hu, hv, z, n and writes h, hu, hv once: 64 B a cell."""
    path = case["path"]
    if path in ("ensemble", "serve"):
        f = [(f["rows"] * f["cols"]) for f in _flows_sizes(case)]
        steps = case["steps"] if path == "ensemble" else 4.0 * case["span"]
        cells = float(sum(f)) * steps
    else:
        cells = float(case["rows"] * case["cols"])
        if path in ("run", "solve", "tangent", "gradient"):
            cells *= case["steps"]
        elif path == "until":
            cells *= 60.0 * case["span"]
    stages = 1 if case.get("integrator") == "euler" else 2
    ops, nbytes = stages * STAGE_OPS + EPILOGUE_OPS, 64.0
    if path == "tangent":  # the values and, per lane, the product rules of every operation
        ops *= 1.0 + 2.0 * case["lanes"]
        nbytes *= 1.0 + case["lanes"]
    elif path == "gradient":  # forward, and its reverse at twice the forward's operations
        ops *= 3.0
        nbytes *= 2.0
    return {"bytes": nbytes * cells, "flops": ops * cells}


def _flows_sizes(case):
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    sides = [case["hi"]] + [int(round(math.exp(lo + (hi - lo) * ((k * 0.61803398875 + 0.1) % 1.0))))
                            for k in range(1, case["count"])]
    return [{"rows": s, "cols": s} for s in sides]


# ------------------------------------------------------------------- exact
def _series(s, t):
    return float(np.interp(t, s[0], s[1]))


def _max0(x):
    return torch.maximum(x, torch.zeros_like(x))


def _safe_div(a, b, ok):
    return torch.where(ok, a / torch.where(ok, b, torch.ones_like(b)), torch.zeros_like(a))


def _safe_sqrt(x, ok):
    return torch.where(ok, torch.sqrt(torch.where(ok, x, torch.ones_like(x))), torch.zeros_like(x))


def _line(k, a, i):
    return a.select(0 if k in (N, S) else 1, i)


def _ghost(f, u, n, side):
    """Ghost state and bed of one side, as vectors along it."""
    kind, val = f["bcs"][side]
    i0, i1 = (0, 1) if side in (N, W) else (-1, -2)
    h, hu, hv = (_line(side, a, i0) for a in u)
    z0 = _line(side, f["z"], i0)
    z = z0 if kind in (OPEN, WALL) else 2.0 * z0 - _line(side, f["z"], i1)
    normal_x = side in (W, E)
    c = torch.full_like(z0, val)
    if kind == WALL:
        hu, hv = (-hu, hv) if normal_x else (hu, -hv)
    elif kind == DISCHARGE:
        hu, hv = (c, hv) if normal_x else (hu, c)
        slope = ((z0 - _line(side, f["z"], i1)) / (f["dx"] if normal_x else f["dy"])).abs()
        dry = (h.detach() < H_DRY) & (slope > 5.0e-4)
        hn = (_line(side, n, i0) * abs(val) / torch.sqrt(torch.where(dry, slope, 1.0))) ** 0.6
        h = torch.where(dry, torch.clamp(hn, max=10.0), h)
    elif kind == DEPTH:
        h = c
    return h, hu, hv, z


def _minmod(a, b):
    pick = torch.where(a.abs() < b.abs(), a, b)
    return torch.where(a * b <= 0.0, torch.zeros_like(a), pick)


def _slopes(p, wet, d):
    """Limited slopes of p along the last axis; zero within two cells of a dry one."""
    out = torch.zeros_like(p)
    n = p.shape[-1]
    if n < 2:
        return out
    dif = (p[..., 1:] - p[..., :-1]) / d
    mid = _minmod(dif[..., :-1], dif[..., 1:]) if n > 2 else dif[..., :0]
    out = torch.cat([dif[..., :1], mid, dif[..., -1:]], -1)
    dry = torch.nn.functional.pad(~wet, (2, 2))
    near = dry[..., :n] | dry[..., 1:n + 1] | dry[..., 2:n + 2] | dry[..., 3:n + 3] | dry[..., 4:n + 4]
    return torch.where(near, torch.zeros_like(out), out)


def _hllc(hl, ql, tl, hr, qr, tr):
    wl, wr = hl > DRY_TOL, hr > DRY_TOL
    cl, cr = _safe_sqrt(G * hl, wl), _safe_sqrt(G * hr, wr)
    ul, ur = _safe_div(ql, hl, wl), _safe_div(qr, hr, wr)
    both = wl & wr
    sl = torch.where(both, torch.minimum(ul - cl, ur - cr), torch.where(wl, ul - cl, ur - 2 * cr))
    sr = torch.where(both, torch.maximum(ul + cl, ur + cr), torch.where(wl, ul + 2 * cl, ur + cr))
    den = hr * (ur - sr) - hl * (ul - sl)
    ok = den.abs() > 1.0e-12
    star = torch.where(ok, _safe_div(hr * (ur - sr) * sl - hl * (ul - sl) * sr, den, ok),
                       0.5 * (sl + sr))
    left = torch.where(sl >= 0, True, torch.where(sr <= 0, False, star >= 0))
    mid = (sl < 0) & (sr > 0)
    h, q, t = (torch.where(left, a, b) for a, b in ((hl, hr), (ql, qr), (tl, tr)))
    u, s, wet = (torch.where(left, a, b) for a, b in ((ul, ur), (sl, sr), (wl, wr)))
    v = _safe_div(t, h, wet)
    zero = torch.zeros_like(h)
    fm = torch.where(wet, q, zero)
    fn = torch.where(wet, q * u + 0.5 * G * h * h, zero)
    ft = torch.where(wet, q * v, zero)
    any_wet = wl | wr
    far = mid & any_wet & (s != star)
    hs = _safe_div(h * (s - u), s - star, far)
    out = (fm + torch.where(far, s * (hs - h), zero),
           fn + torch.where(far, s * (hs * star - q), zero),
           ft + torch.where(far, s * (hs * v - t), zero))
    return [torch.where(any_wet, o, zero) for o in out]


def _faces(z, h, eta, un, ut, raw, wet, d, lo, hi):
    """Fluxes (mass, normal seen by the minus / plus cell, tangential) and
    face beds along the last axis; lo / hi are the ghosts of its two ends and
    raw the (h, normal, tangential momentum) of the state."""
    se, sn, st = (_slopes(a, wet, d) for a in (eta, un, ut))
    zl, zr, wl, wr = z[..., :-1], z[..., 1:], wet[..., :-1], wet[..., 1:]
    zi = torch.where(wl != wr, torch.maximum(zl, zr), 0.5 * (zl + zr))
    zf = torch.cat([0.5 * (lo[3] + z[..., 0])[..., None], zi,
                    0.5 * (z[..., -1] + hi[3])[..., None]], -1)
    k = 0.5 * d
    hm, hp = _max0((eta + k * se)[..., :-1] - zi), _max0((eta - k * se)[..., 1:] - zi)
    um, up = (un + k * sn)[..., :-1], (un - k * sn)[..., 1:]
    vm, vp = (ut + k * st)[..., :-1], (ut - k * st)[..., 1:]

    def join(first, inner, last):
        return torch.cat([first[..., None], inner, last[..., None]], -1)

    left = [join(lo[i], a, raw[i][..., -1]) for i, a in enumerate((hm, hm * um, hm * vm))]
    right = [join(raw[i][..., 0], a, hi[i]) for i, a in enumerate((hp, hp * up, hp * vp))]
    fm, fn, ft = _hllc(left[0], left[1], left[2], right[0], right[1], right[2])
    none = torch.nn.functional.pad(~wl & ~wr, (1, 1))
    fm, fn, ft = (torch.where(none, torch.zeros_like(a), a) for a in (fm, fn, ft))
    return [fm, fn, fn, ft], zf, se


def _stage(f, u, n, dt):
    """One forward-Euler stage in plain tensor operations."""
    h, hu, hv = u
    z, dx, dy = f["z"], f["dx"], f["dy"]
    wet = h.detach() > H_DRY
    fast = h.detach() > H_VEL
    eta, uu, vv = h + z, _safe_div(hu, h, fast), _safe_div(hv, h, fast)
    g = [_ghost(f, u, n, s) for s in (N, S, W, E)]
    X, zx, sx = _faces(z, h, eta, uu, vv, (h, hu, hv), wet, dx, g[W], g[E])
    t = lambda a: a.transpose(0, 1)  # noqa: E731
    swap = lambda q: (q[0], q[2], q[1], q[3])  # noqa: E731
    Y, zy, sy = _faces(t(z), t(h), t(eta), t(vv), t(uu), (t(h), t(hv), t(hu)), t(wet), dy,
                       swap(g[N]), swap(g[S]))
    Y, zy, sy = [t(a) for a in Y], t(zy), t(sy)
    lx, ly = dt / dx, dt / dy
    out = (_max0(X[0][:, 1:]) + _max0(-X[0][:, :-1])) * lx \
        + (_max0(Y[0][1:]) + _max0(-Y[0][:-1])) * ly
    have = _max0(h - H_DRY)
    drain = (out.detach() > have.detach()) & (out.detach() > 0)
    alpha = torch.where(drain, _safe_div(have, out, drain), torch.ones_like(h))

    def scale(F, a, dim):
        m = F[0].detach()
        one = torch.ones_like(a.narrow(dim, 0, 1))
        first = torch.where(m.narrow(dim, 0, 1) < 0, a.narrow(dim, 0, 1), one)
        up = torch.cat([one, a], dim)  # the minus cell's; 1 for flow from outside
        down = torch.cat([first, a.narrow(dim, 1, a.shape[dim] - 1), one], dim)  # the plus cell's
        return [q * torch.where(m > 0, up, down) for q in F]

    X, Y = scale(X, alpha, 1), scale(Y, alpha, 0)
    fx = [a[:, 1:] - a[:, :-1] for a in X]
    fy = [a[1:] - a[:-1] for a in Y]

    def source(eta, slope, zf, d, dim):
        lo = eta - 0.5 * d * slope
        hi = eta + 0.5 * d * slope
        n_ = eta.shape[dim]
        i = torch.arange(n_, device=eta.device).reshape((-1, 1) if dim == 0 else (1, -1))
        lo, hi = torch.where(i > 0, lo, eta), torch.where(i + 1 < n_, hi, eta)
        hl = _max0(lo - zf.narrow(dim, 0, n_))
        hr = _max0(hi - zf.narrow(dim, 1, n_))
        return 0.5 * G * (hl + hr) * ((lo - hl) - (hi - hr)) / d

    e2 = h + z
    s_hu, s_hv = source(e2, sx, zx, dx, 1), source(e2, sy, zy, dy, 0)
    # the two sides of a face see different normal fluxes only by the
    # hydrostatic correction, which is zero with one bed per face up to
    # rounding
    nh = h - (fx[0] * lx + fy[0] * ly)
    keep = nh.detach() > H_VEL
    zero = torch.zeros_like(h)
    nhu = torch.where(fast, hu, zero) - (fx[1] * lx + fy[3] * ly) + s_hu * dt
    nhv = torch.where(fast, hv, zero) - (fx[3] * lx + fy[1] * ly) + s_hv * dt
    dryp = torch.nn.functional.pad(wet, (1, 1, 1, 1), value=True)
    alone = ~wet & ~dryp[:-2, 1:-1] & ~dryp[2:, 1:-1] & ~dryp[1:-1, :-2] & ~dryp[1:-1, 2:]
    keep = keep & ~alone
    return (torch.where(alone, h, torch.where(keep, nh, _max0(nh))),
            torch.where(keep, nhu, zero), torch.where(keep, nhv, zero))


def _speeds(h, hu, hv, cut):
    wet, fast = h > H_DRY, h > cut
    c = _safe_sqrt(G * h, wet)
    sx = torch.where(wet, _safe_div(hu, h, fast).abs() + c, torch.zeros_like(h))
    sy = torch.where(wet, _safe_div(hv, h, fast).abs() + c, torch.zeros_like(h))
    return float(sx.max()), float(sy.max())


def _cfl(f, u, n):
    with torch.no_grad():
        u = [a.detach() for a in u]
        sx, sy = _speeds(*u, H_VEL)
        for s in (N, S, W, E):
            g = _ghost(f, u, n.detach(), s)
            a, b = _speeds(g[0], g[1], g[2], H_DRY)
            sx, sy = max(sx, a), max(sy, b)
        d = sx / f["dx"] + sy / f["dy"]
        return f["cfl"] / d if d > 0 else math.inf


def _euler_or_rk2(f, u, n, dt, rk2):
    v = _stage(f, u, n, dt)
    if not rk2:
        return v
    w = _stage(f, v, n, dt)
    h, hu, hv = ((a + b) * 0.5 for a, b in zip(u, w))
    keep = h.detach() > H_VEL
    zero = torch.zeros_like(h)
    return (torch.where(keep, h, _max0(h)), torch.where(keep, hu, zero),
            torch.where(keep, hv, zero))


def _friction(u, n, dt):
    h, hu, hv = u
    q2 = hu * hu + hv * hv
    on = (h.detach() > H_DRY) & (q2.detach() > 0)
    speed = _safe_div(_safe_sqrt(q2, on), h, on)
    k = 1.0 + dt * G * _safe_div(n * n * speed, torch.where(on, h, torch.ones_like(h)) ** (4 / 3), on)
    return h, hu / k, hv / k


def _forced(f, u, dt, t_new):
    h, hu, hv = u
    if f["rain"] is not None:
        h = h + _series(f["rain"], t_new) * dt
    for r, c, ts, qs in f["src"]:
        add = torch.zeros_like(h)
        add[r, c] = _series((ts, qs), t_new) * dt / (f["dx"] * f["dy"])
        h = h + add
    return h, hu, hv


def _advance(f, u, n, t, steps=None, until=math.inf, each=None, wrap=None):
    """Steps of the whole scheme; returns (u, t, steps taken)."""
    k = 0
    while (steps is None or k < steps) and t < until:
        dt = min(_cfl(f, u, n), 60.0, until - t)

        def one(h, hu, hv, n, dt=dt, t=t):
            v = _friction(_euler_or_rk2(f, (h, hu, hv), n, dt, True), n, dt)
            return _forced(f, v, dt, t + dt)

        u = wrap(one, *u, n) if wrap else one(*u, n)
        t += dt
        k += 1
        if each:
            each(u)
    return u, t, k


def exact(case, seed):
    path = case["path"]
    if path in ("tangent", "gradient"):
        return _exact_derivatives(case, seed)
    with torch.no_grad():
        if path == "ensemble":
            got = [_advance(f, (f["h"], f["hu"], f["hv"]), f["n"], 0.0, case["steps"])
                   for f in _flows(case, seed)]
            return {"left": None, "t": [g[1] for g in got],
                    "u": [g[0][0] if k else g[0] for k, g in enumerate(got)]}
        if path == "serve":
            got = [_advance(f, (f["h"], f["hu"], f["hv"]), f["n"], 0.0, None, f["t_end"])
                   for f in _flows(case, seed)]
            return {"steps": [g[2] for g in got], "u": [g[0] for g in got]}
        f = _flow(case["regime"], case["rows"], case["cols"], seed)
        u, n = (f["h"], f["hu"], f["hv"]), f["n"]
        if path == "free":
            dt = min(_cfl(f, u, n), 60.0)
            v = _friction(_euler_or_rk2(f, u, n, dt, case["integrator"] == "ssprk2"), n, dt)
            return {"dt": dt, "u": _forced(f, v, dt, 0.0)}
        if path == "until":
            u, t, k = _advance(f, u, n, 0.0, None, case["span"])
            return {"t": t, "steps": k, "u": u}
        cells = _gauge_cells(case)
        peak = [float(u[0][r, c]) for r, c in cells]

        def note(v):
            for i, (r, c) in enumerate(cells):
                peak[i] = max(peak[i], float(v[0][r, c]))

        v, t, _ = _advance(f, u, n, 0.0, case.get("steps", 1), each=note if cells else None)
        if path == "step":
            return {"dt": t, "u": v}
        out = {"t": t, "u": v}
        if cells:
            out["peak"] = np.array(peak)
            out["last"] = np.array([float(v[0][r, c]) for r, c in cells])
        return out


def _exact_derivatives(case, seed):
    """Automatic differentiation of the plain scheme (dt held at its value)."""
    f, gauges, obs, zones = _misfit(case, seed)
    dev = f["z"].device
    at = torch.as_tensor(gauges, device=dev)
    want = torch.as_tensor(obs, device=dev)
    u0, n0 = (f["h"], f["hu"], f["hv"]), f["n"]

    def misfit(u, n, wrap):
        terms = []

        def each(v):
            terms.append(((v[0].reshape(-1)[at] - want[len(terms)]) ** 2).sum())

        v, _, _ = _advance(f, u, n, 0.0, case["steps"], each=each, wrap=wrap)
        return torch.stack(terms).sum(), v

    if case["path"] == "gradient":
        from torch.utils.checkpoint import checkpoint
        leaf = [a.clone().requires_grad_(True) for a in (*u0, n0)]
        J, _ = misfit(tuple(leaf[:3]), leaf[3],
                      lambda fn, *a: checkpoint(fn, *a, use_reentrant=False))
        g = torch.autograd.grad(J, leaf)
        return {"J": float(J.detach()), "gn": g[3], "g0": g[:3]}
    import torch.autograd.forward_ad as fwd
    dJ, last = [], []
    for k in range(case["lanes"]):
        with fwd.dual_level():
            zero = torch.zeros_like(n0)
            J, v = misfit(tuple(fwd.make_dual(a, zero) for a in u0),
                          fwd.make_dual(n0, zones[k]), None)
            J = fwd.unpack_dual(J)
            dJ.append(float(J.tangent))
            if k == 0:
                last = [fwd.unpack_dual(a) for a in v]
    lane0 = {d: a.tangent for d, a in zip(("dh", "dhu", "dhv"), last)}
    if case["lanes"] == 1:
        u = dict(lane0, **{d: a.primal for d, a in zip(("h", "hu", "hv"), last)})
        return {"J": float(J.primal), "dJ": dJ[0], "u": u}
    return {"J": float(J.primal), "dJ": np.array(dJ), "lane0": lane0}
