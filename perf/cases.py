"""Workloads of this framework for timing and comparison, through its public
entry points: fire behaviour, propagation (one scenario, batches as CUDA
graphs, the allocation-free entry point, the drop-in over host buffers) and
input preparation.

    listed()             the workloads by name
    draw(rng)            one more of the same ranges
    prepare(case, seed)  what a program holds before the call (device or host inputs, buffers, engine)
    run(state)           one pass; its outputs
    work(case)           bytes and operations a pass cannot do without
    exact(case, seed)    the computed rasters in double precision

Inputs are synthetic: ridged or hilly ground, Voronoi fuel patches with lakes
and roads, smooth wind and per-cell moisture, from the seed.
"""
import ctypes as C
import math
import os
import random
import struct
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "propag-hidalgo_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import py_propag as pp  # noqa: E402
from py_propag import _lib as L  # noqa: E402

F32, F64 = torch.float32, torch.float64
FIRE3 = ("speed_max", "azimuth_max", "eccentricity")


def listed():
    return [
        # one grid a user watches interactively: fire behaviour, then propagation.
        # The smallest call: a kilometre at 8 m, launches and latency only
        {"name": "scenario-128", "kind": "scenario", "width": 128, "height": 128, "ground": "hills",
         "ignitions": 1, "max_time": 21600.0, "tile": 0, "arith": 0, "north_up": False},
        # the plain single scenario: 1024 x 1024, one ignition, ten hours
        {"name": "scenario-1024", "kind": "scenario", "width": 1024, "height": 1024, "ground": "hills",
         "ignitions": 1, "max_time": 36000.0, "tile": 0, "arith": 0, "north_up": False},
        # an oblong north-up map with ragged tiles, in the arithmetic a CPU reproduces
        {"name": "scenario-777x1283", "kind": "scenario", "width": 777, "height": 1283, "ground": "ridges",
         "ignitions": 5, "max_time": 28800.0, "tile": 190, "arith": 1, "north_up": True},
        # the large heterogeneous scenario: 20 km a side, twenty ignitions, twelve hours
        {"name": "scenario-4096", "kind": "scenario", "width": 4096, "height": 4096, "ground": "ridges",
         "ignitions": 20, "max_time": 43200.0, "tile": 0, "arith": 0, "north_up": False},
        # a weather ensemble on shared ground, one CUDA graph for the batch
        {"name": "ensemble-64", "kind": "batch", "jobs": 64, "low": 1024, "high": 1024, "shared": True,
         "max_time": 21600.0},
        # unrelated scenarios of uneven sizes, one CUDA graph for the batch
        {"name": "uneven-32", "kind": "batch", "jobs": 32, "low": 128, "high": 2048, "shared": False,
         "max_time": 36000.0},
        # a process that must not allocate while it serves
        {"name": "static-512", "kind": "static", "width": 512, "height": 512, "ground": "hills",
         "ignitions": 2, "max_time": 21600.0, "tile": 0, "arith": 0, "north_up": False},
        # the drop-in over host arrays: copies in, everything, copies out
        {"name": "host-600x800", "kind": "host", "width": 600, "height": 800, "ground": "ridges",
         "ignitions": 3, "max_time": 14400.0, "tile": 0, "arith": 0, "north_up": False},
        # fire behaviour alone: the three fields a propagation reads, a large map
        {"name": "fire-4096", "kind": "fire", "width": 4096, "height": 4096, "ground": "ridges", "full": False},
        # every field, for a map of intensities and flame lengths
        {"name": "fire-full-1601x1201", "kind": "fire", "width": 1601, "height": 1201, "ground": "ridges",
         "full": True},
        # an hourly forecast: dead fuel moisture from the weather, fused with fire behaviour
        {"name": "weather-1501x1403", "kind": "weather", "width": 1501, "height": 1403, "ground": "ridges",
         "hour": 13, "month": 8},
        # rasters from a DEM and vector layers: slope and aspect, fuel codes, ignition times and list
        {"name": "inputs-3001x2003", "kind": "inputs", "width": 3001, "height": 2003, "polygons": 1200,
         "ignitions": 40},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["scenario", "scenario", "scenario", "batch", "static", "host", "fire", "fire", "weather",
                       "inputs"])
    if kind == "scenario":
        w, h = _log_int(rng, 64, 2600), _log_int(rng, 64, 2600)
        return {"kind": kind, "width": w, "height": h, "ground": rng.choice(["hills", "ridges"]),
                "ignitions": _log_int(rng, 1, 20), "max_time": rng.uniform(3600.0, 43200.0),
                "tile": rng.choice([0, 0, 0, 97, 190, 256]), "arith": rng.choice([0, 0, 0, 1]),
                "north_up": rng.random() < 0.3}
    if kind == "batch":
        shared = rng.random() < 0.5
        low = _log_int(rng, 100, 700)
        return {"kind": kind, "jobs": _log_int(rng, 3, 40), "low": low,
                "high": low if shared else rng.randint(low, 1400), "shared": shared,
                "max_time": rng.uniform(3600.0, 36000.0)}
    if kind == "static":
        return {"kind": kind, "width": _log_int(rng, 64, 1000), "height": _log_int(rng, 64, 1000),
                "ground": rng.choice(["hills", "ridges"]), "ignitions": _log_int(rng, 1, 8),
                "max_time": rng.uniform(3600.0, 21600.0), "tile": rng.choice([0, 128]),
                "arith": rng.choice([0, 0, 1]), "north_up": rng.random() < 0.3}
    if kind == "host":
        return {"kind": kind, "width": _log_int(rng, 64, 1500), "height": _log_int(rng, 64, 1500),
                "ground": rng.choice(["hills", "ridges"]), "ignitions": _log_int(rng, 1, 8),
                "max_time": rng.uniform(3600.0, 21600.0), "tile": 0, "arith": 0, "north_up": rng.random() < 0.3}
    if kind == "fire":
        return {"kind": kind, "width": _log_int(rng, 50, 4000), "height": _log_int(rng, 50, 4000),
                "ground": rng.choice(["hills", "ridges"]), "full": rng.random() < 0.5}
    if kind == "weather":
        return {"kind": kind, "width": _log_int(rng, 100, 1800), "height": _log_int(rng, 100, 1800),
                "ground": rng.choice(["hills", "ridges"]), "hour": rng.randint(0, 23), "month": rng.randint(1, 12)}
    return {"kind": "inputs", "width": _log_int(rng, 200, 4000), "height": _log_int(rng, 200, 4000),
            "polygons": _log_int(rng, 20, 2000), "ignitions": _log_int(rng, 1, 100)}


# ------------------------------------------------------------ synthetic ground ----
DEV = "cuda"
CELL = 5.0  # metres


def _noise(w, h, period, rng):
    """Smooth value noise in [-1, 1], double precision."""
    gw, gh = int(math.ceil(w / period)) + 2, int(math.ceil(h / period)) + 2
    lat = torch.from_numpy(rng.uniform(-1.0, 1.0, (gh, gw))).to(DEV)
    fx = (torch.arange(w, device=DEV, dtype=F64) + 0.5) / period
    fy = (torch.arange(h, device=DEV, dtype=F64) + 0.5) / period
    ix, iy = fx.floor().long(), fy.floor().long()
    tx, ty = fx - ix, fy - iy
    sx, sy = (tx * tx * (3 - 2 * tx))[None, :], (ty * ty * (3 - 2 * ty))[:, None]
    a, b = lat[iy][:, ix], lat[iy][:, ix + 1]
    c, d = lat[iy + 1][:, ix], lat[iy + 1][:, ix + 1]
    return (a + (b - a) * sx) * (1 - sy) + (c + (d - c) * sx) * sy


def _dem(w, h, ground, rng):
    if ground == "hills":  # Gaussian hills up to 800 m
        k = 30
        x = (torch.arange(w, device=DEV, dtype=F64) + 0.5) * CELL
        y = (torch.arange(h, device=DEV, dtype=F64) + 0.5) * CELL
        cx, cy, sig, top = (torch.from_numpy(v).to(DEV) for v in (
            rng.uniform(0, w * CELL, k), rng.uniform(0, h * CELL, k), rng.uniform(150.0, 1500.0, k),
            rng.uniform(0.2, 1.0, k)))
        gx = torch.exp(-0.5 * ((x[None, :] - cx[:, None]) / sig[:, None]) ** 2)
        gy = torch.exp(-0.5 * ((y[None, :] - cy[:, None]) / sig[:, None]) ** 2) * top[:, None]
        z = gy.T @ gx
        z -= z.min()
        return z * (800.0 / float(z.max().clamp_min(1e-9)))
    z, amp, period = torch.zeros((h, w), device=DEV, dtype=F64), 1.0, max(w, h) / 4.0
    for _ in range(6):  # ridges, steepest slope 45 degrees
        if period < 2:
            break
        r = 1.0 - _noise(w, h, period, rng).abs()
        z += amp * r * r
        amp, period = amp * 0.5, period / 2.0
    s, _ = _slope_aspect(z)
    return z / float(s.max().clamp_min(1e-9))


def _gradient(z, step, dim):
    g = torch.zeros_like(z)
    n = z.shape[dim]
    if n > 1:
        g.narrow(dim, 1, n - 2).copy_((z.narrow(dim, 2, n - 2) - z.narrow(dim, 0, n - 2)) / (2.0 * step))
        g.narrow(dim, 0, 1).copy_((z.narrow(dim, 1, 1) - z.narrow(dim, 0, 1)) / step)
        g.narrow(dim, n - 1, 1).copy_((z.narrow(dim, n - 1, 1) - z.narrow(dim, n - 2, 1)) / step)
    return g


def _slope_aspect(z):
    """Rise over run, and the compass azimuth of the downhill direction."""
    gx, gy = _gradient(z, CELL, 1), _gradient(z, CELL, 0)
    s = torch.hypot(gx, gy)
    a = torch.atan2(-gx, -gy)
    a = torch.where(a < 0, a + 2 * math.pi, a)
    return s, torch.where(s == 0, torch.zeros_like(a), a)


def _fuel(w, h, ground, rng):
    """Voronoi patches of models 1..13 about 64 cells wide, with patches
    (hills) or lakes and roads (ridges) that do not burn."""
    g = 64.0
    gw, gh = int(w / g) + 3, int(h / g) + 3
    px, py = (torch.from_numpy(rng.uniform(0, g, (gh, gw))).to(DEV, F32) for _ in range(2))
    code = rng.integers(1, 14, (gh, gw))
    if ground == "hills":
        code[rng.uniform(size=(gh, gw)) < 0.05] = 0
    code = torch.from_numpy(code.astype(np.uint8)).to(DEV)
    x = (torch.arange(w, device=DEV, dtype=F32) + 0.5)[None, :].expand(h, w)
    y = (torch.arange(h, device=DEV, dtype=F32) + 0.5)[:, None].expand(h, w)
    bx, by = (x / g).long(), (y / g).long()
    best = torch.full((h, w), 1e30, device=DEV, dtype=F32)
    fuel = torch.zeros((h, w), device=DEV, dtype=torch.uint8)
    for j in range(3):
        for i in range(3):  # seeds of the lattice cells around (shifted by one: index 0 lies outside the map)
            sx = px[by + j, bx + i] + (bx + (i - 1)) * g
            sy = py[by + j, bx + i] + (by + (j - 1)) * g
            d = (x - sx) ** 2 + (y - sy) ** 2
            near = d < best
            best = torch.where(near, d, best)
            fuel = torch.where(near, code[by + j, bx + i], fuel)
    if ground == "ridges":
        big = max(w, h)
        covered = 0.0
        while covered < 0.1 * w * h:  # lakes
            r = rng.uniform(0.01, 0.05) * big
            cx, cy = rng.uniform(0, w), rng.uniform(0, h)
            x0, x1 = max(int(cx - r), 0), min(int(cx + r) + 2, w)
            y0, y1 = max(int(cy - r), 0), min(int(cy + r) + 2, h)
            lake = (x[y0:y1, x0:x1] - cx) ** 2 + (y[y0:y1, x0:x1] - cy) ** 2 <= r * r
            fuel[y0:y1, x0:x1][lake] = 0
            covered += 0.8 * math.pi * r * r
        for _ in range(max(2, round(6 * big / 4096))):  # roads, two to three cells wide
            ax, ay, t = rng.uniform(0, w), rng.uniform(0, h), rng.uniform(0, 2 * math.pi)
            for _seg in range(6):
                t += rng.normal(0, 0.5)
                n = rng.uniform(0.1, 0.3) * big
                ex, ey = ax + n * math.sin(t), ay + n * math.cos(t)
                x0, x1 = max(int(min(ax, ex)) - 2, 0), min(int(max(ax, ex)) + 3, w)
                y0, y1 = max(int(min(ay, ey)) - 2, 0), min(int(max(ay, ey)) + 3, h)
                if x0 < x1 and y0 < y1:
                    q = (x[y0:y1, x0:x1] - ax) * math.cos(t) - (y[y0:y1, x0:x1] - ay) * math.sin(t)
                    fuel[y0:y1, x0:x1][q.abs() <= 1.25] = 0
                ax, ay = ex, ey
    return fuel


def _terrain(w, h, ground, rng, gen):
    slope, aspect = _slope_aspect(_dem(w, h, ground, rng))
    t = {"fuel_code": _fuel(w, h, ground, rng), "slope": slope.to(F32), "aspect": aspect.to(F32)}
    moist = (("d1hr", 0.06), ("d10hr", 0.07), ("d100hr", 0.08), ("herb", 0.60), ("wood", 0.90))
    if ground == "hills":  # one wind and one moisture for the map
        speed, to = math.exp(math.log(6.0) + 0.3 * rng.standard_normal()), 45.0 + rng.uniform(-30.0, 30.0)
        t["wind_speed"] = torch.full((h, w), speed, device=DEV, dtype=F32)
        t["wind_azimuth"] = torch.full((h, w), math.radians(to), device=DEV, dtype=F32)
        for k, v in moist:
            t[k] = torch.full((h, w), v, device=DEV, dtype=F32)
    else:
        big = max(w, h)
        t["wind_speed"] = (7.5 + 7.5 * _noise(w, h, big / 3.0, rng)).clamp(0.0, 15.0).to(F32)
        t["wind_azimuth"] = torch.remainder(math.radians(45.0) + math.radians(60.0) * _noise(w, h, big / 3.0, rng),
                                            2 * math.pi).to(F32)
        for k, v in moist:
            t[k] = v + 0.04 * (torch.rand((h, w), device=DEV, generator=gen, dtype=F32) - 0.5)
    return {k: v.contiguous().view(-1) for k, v in t.items()}


def _rngs(seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    return np.random.default_rng(int(seed)), gen


def _ignitions(fuel, w, h, count, rng, spread=0.0):
    """Burnable cells; times 0, or staggered over `spread` seconds."""
    f = fuel.view(h, w).cpu().numpy()
    out = []
    for _ in range(200 * count):
        if len(out) == count:
            break
        x, y = int(rng.integers(0, w)), int(rng.integers(0, h))
        if f[y, x] != 0:
            out.append((x, y, float(rng.uniform(0.0, spread)) if out and spread else 0.0))
    return out


def _ignition_array(ign):
    a = np.array(ign, dtype=[("x", "<u4"), ("y", "<u4"), ("t", "<f4")])
    return torch.from_numpy(np.frombuffer(a.tobytes() or bytes(12), np.uint8).copy()).to(DEV), len(a)


def _ptrs(t):
    return L.PropagTerrainPtrs(*[t[k].data_ptr() if k in t else None for k in L.TERRAIN_FIELDS])


def _results(n):
    b = {k: torch.zeros(n, dtype=F32, device=DEV) for k in FIRE3 + ("time",)}
    b["refs_x"] = torch.zeros(n, dtype=torch.int16, device=DEV)
    b["refs_y"] = torch.zeros(n, dtype=torch.int16, device=DEV)
    b["boundaries"] = torch.zeros((n + 31) // 32, dtype=torch.int32, device=DEV)
    return b


def _job(w, h, t, ign, case, b, cell=CELL):
    """A job over device buffers `b`, and what it keeps alive."""
    ign_d, k = _ignition_array(ign)
    j = L.PropagJob()
    j.width, j.height, j.dx, j.dy = w, h, cell, -cell if case.get("north_up") else cell
    j.max_time, j.tile, j.arith = case["max_time"], case.get("tile", 0), case.get("arith", 0)
    j.ignitions, j.n_ignitions = ign_d.data_ptr(), k
    for name, v in b.items():
        setattr(j, name, v.data_ptr())
    return j, (t, ign_d)


def _check(rc, what):
    if rc != 0:
        raise RuntimeError("%s: %s" % (what, L.last_error()))


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


# ------------------------------------------------------------------- the passes ----
def prepare(case, seed):
    rng, gen = _rngs(seed)
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, rng, gen)
    w, h = case["width"], case["height"]
    if kind == "inputs":
        return _prepare_inputs(case, rng)
    t = _terrain(w, h, case["ground"], rng, gen)
    state = {"kind": kind, "case": case, "n": w * h, "terrain": t, "ptrs": _ptrs(t)}
    if kind == "fire":
        names = L.FIRE_FIELDS if case["full"] else FIRE3
        state["out"] = {k: torch.zeros(w * h, dtype=F32, device=DEV) for k in names}
        if case["full"]:
            state["fields"] = L.PropagFireFields(*[state["out"][k].data_ptr() for k in L.FIRE_FIELDS])
    elif kind == "weather":
        state["weather"] = _weather(w * h, gen)
        state["wptrs"] = L.PropagWeatherPtrs(*[v.data_ptr() for v in state["weather"].values()])
        state["out"] = {k: torch.zeros(w * h, dtype=F32, device=DEV) for k in FIRE3}
    elif kind == "host":
        state["ign"] = _ignitions(t["fuel_code"], w, h, case["ignitions"], rng)
        state["host"] = {k: v.cpu().numpy().reshape(h, w) for k, v in t.items()}
        d = -CELL if case["north_up"] else CELL
        gt = [0.0, CELL, 0.0, 0.0 if d > 0 else h * CELL, 0.0, d]
        g = pp.PyGeoReference(w, h, "+proj=utm +zone=30 +ellps=GRS80 +units=m +no_defs", gt)
        state["settings"] = pp.PySettings(g, case["max_time"])
        del state["terrain"], state["ptrs"]
    else:
        ign = _ignitions(t["fuel_code"], w, h, case["ignitions"], rng, spread=1800.0)
        state["out"] = _results(w * h)
        state["job"], state["keep"] = _job(w, h, t, ign, case, state["out"])
        if kind == "scenario":
            state["engine"] = pp.Engine()
    return state


def _prepare_batch(case, rng, gen):
    # sides evenly spread over their logarithm, in an order of no use to a queue
    k, ratio = case["jobs"], case["high"] / case["low"]
    sizes = [int(round(case["low"] * ratio ** ((i * 0.618034) % 1.0))) for i in range(1, k)] + [case["high"]]
    # every member's buffers in one allocation per raster, members 256-byte aligned
    room = [(s * s + 2047) // 2048 * 2048 for s in sizes]
    flat = _results(sum(room))
    jobs, ptrs, keep, at = [], [], [], 0
    shared = _terrain(sizes[0], sizes[0], "hills", rng, gen) if case["shared"] else None
    for side, pad in zip(sizes, room):
        n = side * side
        if case["shared"]:
            t = dict(shared)
            speed, to = math.exp(math.log(6.0) + 0.3 * rng.standard_normal()), 45.0 + rng.uniform(-30.0, 30.0)
            t["wind_speed"] = torch.full((n,), speed, device=DEV, dtype=F32)
            t["wind_azimuth"] = torch.full((n,), math.radians(to), device=DEV, dtype=F32)
            off = float(rng.uniform(-0.02, 0.02))
            for k in ("d1hr", "d10hr", "d100hr"):
                t[k] = shared[k] + off
            count, cell, limit = 1, CELL, case["max_time"]
        else:
            t = _terrain(side, side, "hills", rng, gen)
            count, cell = int(rng.integers(1, 11)), float(rng.uniform(5.0, 30.0))
            limit = float(rng.uniform(0.1, 1.0)) * case["max_time"]
        ign = _ignitions(t["fuel_code"], side, side, count, rng)
        b = {k: v[at // 32:] if k == "boundaries" else v[at:] for k, v in flat.items()}
        j, k = _job(side, side, t, ign, {"max_time": limit}, b, cell)
        jobs.append(j)
        ptrs.append(_ptrs(t))
        keep.append(k)
        at += pad
    torch.cuda.synchronize()  # the graph is sized on a stream of its own
    return {"kind": "batch", "graph": pp.Graph(jobs, ptrs), "out": flat, "keep": keep}


def _weather(n, gen):
    def u(k, low, high):
        return low + (high - low) * torch.rand((k, n), device=DEV, generator=gen, dtype=F32)
    rain = u(6, -30.0, 12.0).clamp_min(0.0)  # most days dry
    return {"temperature": u(24, 2.0, 40.0), "humidity": u(24, 8.0, 98.0), "cloud_cover": u(24, 0.0, 100.0),
            "precipitation": rain}


def _wkb_polygon(rings):
    return struct.pack("<BII", 1, 3, len(rings)) + b"".join(
        struct.pack("<I", len(r)) + np.asarray(r, "<f8").tobytes() for r in rings)


def _wkb_line(pts):
    return struct.pack("<BII", 1, 2, len(pts)) + np.asarray(pts, "<f8").tobytes()


def _features(kind, items):
    """A C array of features over WKB buffers, and the buffers."""
    arr, keep = (kind * len(items))(), []
    for i, (value, wkb) in enumerate(items):
        b = (C.c_uint8 * len(wkb)).from_buffer_copy(wkb)
        keep.append(b)
        setattr(arr[i], "code" if kind is L.FFIFuelFeature else "time", value)
        arr[i].geom_wkb, arr[i].geom_wkb_len = C.cast(b, C.POINTER(C.c_uint8)), len(wkb)
    return arr, keep


def _blob(cx, cy, r, k, rng):
    a = np.sort(rng.uniform(0, 2 * np.pi, k))
    q = r * rng.uniform(0.5, 1.0, k)
    p = np.stack([cx + q * np.cos(a), cy + q * np.sin(a)], 1)
    return np.concatenate([p, p[:1]])


def _prepare_inputs(case, rng):
    w, h = case["width"], case["height"]
    W, H = w * CELL, h * CELL
    proj = "+proj=utm +zone=30 +ellps=GRS80 +units=m +no_defs"
    g = pp.PySettings(pp.PyGeoReference(w, h, proj, [0.0, CELL, 0.0, 0.0, 0.0, CELL]), 3600.0).inner.geo_ref
    fuels, times = [], []
    for _ in range(case["polygons"]):
        r = math.exp(rng.uniform(math.log(10 * CELL), math.log(0.08 * max(W, H))))
        fuels.append((int(rng.integers(0, 14)),
                      _wkb_polygon([_blob(rng.uniform(0, W), rng.uniform(0, H), r, int(rng.integers(5, 60)), rng)])))
    for i in range(case["ignitions"]):
        x, y = rng.uniform(0, W), rng.uniform(0, H)
        if i % 3 == 0:
            wkb = struct.pack("<BIdd", 1, 1, x, y)
        elif i % 3 == 1:
            wkb = _wkb_line(np.stack([x + np.cumsum(rng.normal(0, 20 * CELL, 12)),
                                      y + np.cumsum(rng.normal(0, 20 * CELL, 12))], 1))
        else:
            wkb = _wkb_polygon([_blob(x, y, 15 * CELL, 9, rng)])
        times.append((float(rng.uniform(0.0, 7200.0)), wkb))
    farr, fkeep = _features(L.FFIFuelFeature, fuels)
    tarr, tkeep = _features(L.FFITimeFeature, times)
    n, most = w * h, min(w * h, 200 * 1000)
    out = {"slope": torch.zeros(n, dtype=F32, device=DEV), "aspect": torch.zeros(n, dtype=F32, device=DEV),
           "fuel": torch.zeros(n, dtype=torch.uint8, device=DEV), "times": torch.zeros(n, dtype=F32, device=DEV),
           "ignitions": torch.zeros(3 * most, dtype=torch.int32, device=DEV)}
    return {"kind": "inputs", "w": w, "h": h, "dem": _dem(w, h, "ridges", rng).mul(400.0).to(F32).contiguous(),
            "geo": g, "crs": proj.encode(), "fuels": (farr, len(fuels)), "times": (tarr, len(times)),
            "keep": (fkeep, tkeep), "most": most, "out": out}


def run(state):
    lib, s, kind = L.lib(), _stream(), state["kind"]
    if kind == "batch":
        state["graph"].launch(torch.cuda.current_stream().cuda_stream)
        return state["out"]
    if kind == "host":
        r = pp.propagate_arrays(state["settings"], state["host"], state["ign"])
        return {"time": r.arrival_times, "refs_x": r.refs_x.view(np.int16), "refs_y": r.refs_y.view(np.int16),
                "boundaries": r.boundary_change.view(np.int32)}
    if kind == "inputs":
        o, w, h, g = state["out"], state["w"], state["h"], state["geo"]
        _check(lib.propag_slope_aspect_device(w, h, CELL, CELL, state["dem"].data_ptr(), o["slope"].data_ptr(),
                                              o["aspect"].data_ptr(), s), "slope_aspect")
        _check(lib.propag_rasterize_fuels_device(state["fuels"][0], state["fuels"][1], state["crs"], C.byref(g),
                                                 o["fuel"].data_ptr(), s), "rasterize_fuels")
        _check(lib.propag_rasterize_times_device(C.byref(g), state["times"][0], state["times"][1],
                                                 o["times"].data_ptr(), s), "rasterize_times")
        count = lib.propag_ignitions_from_times_device(o["times"].data_ptr(), w, h, o["ignitions"].data_ptr(),
                                                       state["most"], s)
        if count < 0:
            raise RuntimeError("ignitions_from_times: " + L.last_error())
        return {**o, "count": int(count)}
    o = state["out"]
    if kind == "weather":
        c = state["case"]
        _check(lib.propag_fire_weather_device(state["n"], c["hour"], c["month"], C.byref(state["wptrs"]),
                                              C.byref(state["ptrs"]), *[o[k].data_ptr() for k in FIRE3], s),
               "fire_weather")
        return o
    if kind == "fire" and state["case"]["full"]:
        _check(lib.propag_fire_full_device(state["n"], C.byref(state["ptrs"]), C.byref(state["fields"]), s),
               "fire_full")
        return o
    _check(lib.propag_fire_simple_device(state["n"], C.byref(state["ptrs"]), *[o[k].data_ptr() for k in FIRE3], s),
           "fire_simple")
    if kind == "scenario":
        state["engine"].run([state["job"]], stream=torch.cuda.current_stream().cuda_stream, want_stats=False)
    elif kind == "static":
        _check(lib.propag_run_device_static(C.byref(state["job"]), s, None), "run_device_static")
    return o


# ------------------------------------------------------------------------ work ----
def work(case):
    kind = case["kind"]
    if kind == "batch":
        side = case["low"] if case["shared"] else (case["low"] * case["high"]) ** 0.5
        n = case["jobs"] * side * side
        return {"bytes": n * (37 + 12 + 8.125), "flops": n * 900.0}
    n = case["width"] * case["height"]
    if kind == "fire":
        return {"bytes": n * (37 + (40 if case["full"] else 12)), "flops": n * 250.0}
    if kind == "weather":
        return {"bytes": n * (85 + 12), "flops": n * 450.0}
    if kind == "inputs":  # DEM in, slope and aspect out, a code, a time
        return {"bytes": n * (4 + 8 + 1 + 4), "flops": n * 60.0}
    # terrain in; fire rasters, times, references and boundary bits out
    return {"bytes": n * (37 + (12 if kind != "host" else 0) + 8.125), "flops": n * 900.0}


# ----------------------------------------------------- double-precision values ----
# The standard fuel models: bed depth (ft), moisture of extinction, particles
# (class, load lb/ft2, surface-to-volume 1/ft); class d: dead, h: herbaceous, w: woody.
_MODELS = [
    None,
    (1.0, 0.12, "d 0.034 3500"),
    (1.0, 0.15, "d 0.092 3000, d 0.046 109, d 0.023 30, h 0.023 1500"),
    (2.5, 0.25, "d 0.138 1500"),
    (6.0, 0.20, "d 0.230 2000, d 0.184 109, d 0.092 30, w 0.230 1500"),
    (2.0, 0.20, "d 0.046 2000, d 0.023 109, w 0.092 1500"),
    (2.5, 0.25, "d 0.069 1750, d 0.115 109, d 0.092 30"),
    (2.5, 0.40, "d 0.052 1750, d 0.086 109, d 0.069 30, w 0.017 1550"),
    (0.2, 0.30, "d 0.069 2000, d 0.046 109, d 0.115 30"),
    (0.2, 0.25, "d 0.134 2500, d 0.019 109, d 0.007 30"),
    (1.0, 0.25, "d 0.138 2000, d 0.092 109, d 0.230 30, w 0.092 1500"),
    (1.0, 0.15, "d 0.069 1500, d 0.207 109, d 0.253 30"),
    (2.3, 0.20, "d 0.184 1500, d 0.644 109, d 0.759 30"),
    (3.0, 0.25, "d 0.322 1500, d 0.058 109, d 1.288 30"),
]


def _size_class(savr):
    return sum(savr <= v for v in (1200.0, 192.0, 96.0, 48.0, 16.0))


def _burn64(code, t):
    """Rothermel's surface fire of one fuel model, SI units, all in float64
    (t: the cells' inputs); the ten fields by name."""
    depth, mext, text = _MODELS[code]
    parts = []
    for p in text.split(","):
        c, load, savr = p.split()
        load, savr = float(load), float(savr)
        m = "herb" if c == "h" else "wood" if c == "w" else ("d1hr", "d1hr", "d10hr", "d10hr", "d100hr",
                                                            "d100hr")[_size_class(savr)]
        parts.append({"live": c != "d", "load": load, "savr": savr, "area": load * savr / 32.0, "m": m,
                      "size": _size_class(savr), "eps": math.exp(-138.0 / savr)})
    whole = sum(p["area"] for p in parts)
    life = {}
    for live in (False, True):
        mine = [p for p in parts if p["live"] == live]
        area = sum(p["area"] for p in mine)
        for p in mine:
            p["aw"] = p["area"] / area
        for p in mine:
            p["sw"] = sum(q["aw"] for q in mine if q["size"] == p["size"])
        life[live] = {"w": area / whole, "savr": sum(p["aw"] * p["savr"] for p in mine),
                      "load": sum(p["sw"] * p["load"] * (1.0 - 0.0555) for p in mine),
                      "eta_s": min(1.0, 0.174 / 0.01 ** 0.19) if mine else 1.0, "parts": mine}
    sigma = sum(v["w"] * v["savr"] for v in life.values())
    bulk = sum(p["load"] for p in parts) / depth
    beta = bulk / 32.0
    ratio = beta / (3.348 * sigma ** -0.8189)
    flux = math.exp((0.792 + 0.681 * math.sqrt(sigma)) * (beta + 0.1)) / (192.0 + 0.2595 * sigma)
    aa = 133.0 * sigma ** -0.7913
    gamma = sigma ** 1.5 / (495.0 + 0.0594 * sigma ** 1.5) * ratio ** aa * math.exp(aa * (1.0 - ratio))
    slope_k = 5.275 * beta ** -0.3
    wind_b = 0.02526 * sigma ** 0.54
    c, e = 7.47 * math.exp(-0.133 * sigma ** 0.55), 0.715 * math.exp(-0.000359 * sigma)
    wind_k, wind_e = c * ratio ** -e, ratio ** e / c
    residence = 384.0 / sigma

    def damping(moist, limit):
        r = moist / limit
        v = 1.0 - 2.59 * r + 5.11 * r * r - 3.52 * r ** 3
        return torch.where(moist >= limit, torch.zeros_like(v), v)

    dead, live = life[False]["parts"], life[True]["parts"]
    rbqig = bulk * sum((250.0 + 1116.0 * t[p["m"]]) * p["aw"] * life[p["live"]]["w"] * p["eps"] for p in parts)
    limit = torch.full_like(rbqig, mext)
    rx = life[False]["load"] * 8000.0 * life[False]["eta_s"] * gamma * damping(
        sum(p["aw"] * t[p["m"]] for p in dead), limit)
    if live:
        fine = sum(p["load"] * p["eps"] for p in dead)
        moist = sum(t[p["m"]] * p["eps"] * p["load"] for p in dead) / fine
        wet = 2.9 * fine / sum(p["load"] * math.exp(-500.0 / p["savr"]) for p in live)
        wet = (wet * (1.0 - moist / mext) - 0.226).clamp_min(mext)
        rx = rx + life[True]["load"] * 8000.0 * life[True]["eta_s"] * gamma * damping(
            sum(p["aw"] * t[p["m"]] for p in live), wet)
    speed0 = rx * flux / rbqig
    foot, btu, tiny = 0.3048, 1054.35, 1e-6
    slope, wind, waz, aspect = t["slope"], t["wind_speed"], t["wind_azimuth"], t["aspect"]
    fpm = wind / (foot / 60.0)
    phi_s, phi_w = slope_k * slope * slope, wind_k * fpm ** wind_b
    phi = phi_s + phi_w
    up = torch.where(aspect >= math.pi, aspect - math.pi, aspect + math.pi)
    # the wind's push across the slope, as vectors in units of speed0
    split = torch.where(up <= waz, waz - up, 2 * math.pi - up + waz)
    x, y = phi_s + phi_w * torch.cos(split), phi_w * torch.sin(split)
    both = torch.hypot(x, y)
    turn = torch.atan2(y, x)
    az = up + torch.where(turn < 0, turn + 2 * math.pi, turn)
    az = torch.where(az > 2 * math.pi, az - 2 * math.pi, az)
    zero = torch.zeros_like(phi)
    flat, calm = slope < tiny, (wind < tiny) | ((up - waz).abs() < tiny)
    pew = torch.where(flat | calm, phi, both)
    ew = torch.where(flat, fpm, (pew * wind_e) ** (1.0 / wind_b))
    az = torch.where(flat, waz, torch.where(calm, up, az))
    still, none = phi < tiny, speed0 < tiny
    pew = torch.where(still | none, phi, pew)
    ew, az = torch.where(still | none, zero, ew), torch.where(still | none, zero, az)
    top = 0.9 * rx
    over = (ew > top) & ~still & ~none
    pew = torch.where(over, wind_k * top ** wind_b, pew)
    ew = torch.where(over, top, ew)
    smax = torch.where(none, zero, torch.where(still, speed0, speed0 * (1.0 + pew)))
    lw = 1.0 + 0.002840909 * ew
    byrams = residence * smax * rx / 60.0
    flame = torch.where(byrams > tiny, 0.45 * byrams.clamp_min(tiny) ** 0.46, zero)
    return {"rx_int": rx * (btu / foot ** 2 / 60.0), "speed0": speed0 * (foot / 60.0),
            "hpua": rx * residence * (btu / foot ** 2), "phi_eff_wind": pew, "speed_max": smax * (foot / 60.0),
            "azimuth_max": az, "eccentricity": torch.sqrt(lw * lw - 1.0) / lw,
            "residence_time": torch.full_like(rx, residence * 60.0), "byrams_max": byrams * (btu / foot),
            "flame_max": flame * foot}


def exact(case, seed):
    """Fire behaviour, slope and aspect in float64.  Arrival times depend on
    the order in which cells adopt their neighbours' references, down to the
    last bit of a float: they have no value in another precision.  Dead fuel
    moisture is a chain of table look-ups and thresholds in float, and rasters
    of codes and ignition times are picked, not computed."""
    kind = case["kind"]
    if kind in ("batch", "host", "weather"):
        return None
    state = prepare({**case, "kind": "fire", "full": False} if kind in ("scenario", "static") else case, seed)
    if kind == "inputs":
        s, a = _slope_aspect(state["dem"].double())
        return {"slope": s.view(-1), "aspect": a.view(-1), "fuel": None, "times": None, "ignitions": None,
                "count": None}
    names = L.FIRE_FIELDS if kind == "fire" and case["full"] else FIRE3
    out = {k: torch.zeros(state["n"], dtype=F64, device=DEV) for k in names}
    for code in range(1, 14):
        at = (state["terrain"]["fuel_code"] == code).nonzero().view(-1)
        for part in at.split(1 << 22):
            v = _burn64(code, {k: x[part].double() for k, x in state["terrain"].items() if k != "fuel_code"})
            for k in names:
                out[k][part] = v[k]
    if kind in ("scenario", "static"):
        out.update({"time": None, "refs_x": None, "refs_y": None, "boundaries": None})
    return out


if __name__ == "__main__":
    for c in listed() + [draw(random.Random(i)) for i in range(3)]:
        print(c, work(c))
