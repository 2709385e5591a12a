"""The work that programs give this framework, as cases to be timed: travel-time fields one at a time
and in batches, whole forward steps, rays on tables that a program already has, event location, LSQR
on the rows of a ray call, and a burst of requests to the serving loop. Every case goes through the
package's public entry points and takes its results the way a program does (host arrays).

Case kinds and their ranges (`listed` holds the named sizes, `draw` others of the same ranges):

  solve    EikonalCuda.solve: 1-30 sources on one grid of 12-161 nodes per axis, FP64 or FP32, the
           reference's rule ("engine") or the throughput rule ("fast"), double or float output
  tables   location.Tables.build: P and S tables of 1-10 stations (161x161x81 and below)
  multi    EikonalCuda.solve_multi: 4-24 grids of uneven size, half of them with growing depth steps
  forward  RayKernels.compute: tables of every (station, phase) and the CSR rows of the arrivals
  rays     rays.trace_rows on given tables: 50-40,000 rays
  locate   location.locate: 20-600 events on resident tables
  lsqr     lsqr.solve_rows on the rows of a ray call
  serve    Server: 4-24 mixed requests submitted together and waited for
"""
from __future__ import annotations

import ctypes as C
import functools
import math
import random

import numpy as np
import torch

from tomostar_b200 import _lib as L
from tomostar_b200 import location, lsqr, rays
from tomostar_b200.eikonal import EikonalCuda, point_source
from tomostar_b200.grid import DEG2RAD, EARTH_RADIUS_KM, GridDef
from tomostar_b200.serving import Server
from tomostar_b200.synthetic import km_to_geo, regular_grid

DEVICE = "cuda"
MODES = {"engine": L.MODE_ENGINE, "fast": L.MODE_FAST}


# ---- cases -------------------------------------------------------------------------------------------

def listed() -> list[dict]:
    return [
        # One source on the reference's self-test grid: the smallest call a host makes (try_create's
        # gate, a quick look at one station), all latency.
        dict(name="solve_one_22x20x16", kind="solve", nx=22, ny=20, nz=16, h=1.0, fields=1, prec=64, mode="engine",
             out=64),
        # One source on the 61x61x31 model with the reference's rule and FP64 output (TrySolve as the
        # C# host calls it for one station).
        dict(name="solve_one_61x61x31", kind="solve", nx=61, ny=61, nz=31, h=1.0, fields=1, prec=64, mode="engine",
             out=64),
        # A resolution test's batch: 25 sources on an 81x81x41 checkerboard, float tables wanted.
        dict(name="solve_25_81x81x41_fast", kind="solve", nx=81, ny=81, nz=41, h=1.0, fields=25, prec=64,
             mode="fast", out=32),
        # The tables a relocation starts from: 5 stations, P and S, bitwise mode, 161x161x81.
        dict(name="tables_10_161x161x81", kind="tables", nx=161, ny=161, nz=81, h=0.5, stations=5, prec=64),
        # Sources each on its own grid, half with variable depth spacing, in one launch; the paired
        # FP32 precision with the tile shape and scheduler the autotuner picks for such batches.
        dict(name="multi_16_uneven_f32", kind="multi", grids=16, scale=0.7, prec=32, mode="fast", tile=1, scheduler=1),
        # The forward step of one inversion iteration: 25 stations x P, S on 121x121x61, 7,500 rays.
        dict(name="forward_50_121x121x61", kind="forward", nx=121, nz=61, h=0.5, stations=25, events=150, rays=7500,
             prec=64, tile=6, scheduler=1),
        # The same step at an earlier stage of a project: few stations, default settings, FP32.
        dict(name="forward_8_97x97x49_f32", kind="forward", nx=97, nz=49, h=0.5, stations=4, events=60, rays=480,
             prec=32, tile=0, scheduler=0),
        # The largest: a share of the regional step (401x401x121 at 0.25 km), 12 stations x P, S and
        # 45,000 rays, with the tile shape documented for large uniform batches.
        dict(name="forward_24_401x401x121", kind="forward", nx=401, nz=121, h=0.25, stations=12, events=2500,
             rays=45000, prec=64, tile=6, scheduler=0),
        # A station's new picks traced on its tables: few rays.
        dict(name="rays_400_121x121x61", kind="rays", nx=121, nz=61, h=0.5, tables=6, rays=400),
        # A relocation of 400 events on 60 resident tables of 161x161x81 nodes.
        dict(name="locate_400_161x161x81", kind="locate", nx=161, nz=81, h=0.5, stations=30, events=400, share=0.8),
        # The inversion's linear solve on 12,000 rows that a ray call left on the device: the first 12 iterations
        # (beyond them the bidiagonalisation amplifies rounding and no two summation orders agree).
        dict(name="lsqr_12000_rows_121x121x61", kind="lsqr", nx=121, nz=61, h=0.5, tables=20, rays=12000, iterations=12),
        # The serving loop under a burst: 20 requests of the three sorts of the serving load at once.
        dict(name="serve_burst_20", kind="serve", requests=20, prec=64),
    ]


def _log(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["solve", "solve", "solve", "tables", "multi", "forward", "forward", "rays", "rays", "locate",
                       "lsqr", "serve"])
    if kind == "solve":
        return dict(kind=kind, nx=_log(rng, 12, 161), ny=_log(rng, 12, 161), nz=_log(rng, 8, 81),
                    h=round(rng.uniform(0.25, 2.0), 2), fields=_log(rng, 1, 30), prec=rng.choice([64, 64, 32]),
                    mode=rng.choice(["engine", "fast"]), out=rng.choice([64, 32]))
    if kind == "tables":
        return dict(kind=kind, nx=_log(rng, 21, 161), ny=_log(rng, 21, 161), nz=_log(rng, 17, 81),
                    h=round(rng.uniform(0.5, 2.5), 2), stations=_log(rng, 1, 10), prec=rng.choice([64, 64, 32]))
    if kind == "multi":
        tile, sched = rng.choice([(1, 1), (1, 1), (0, 0), (6, 1)])
        return dict(kind=kind, grids=_log(rng, 4, 24), scale=round(rng.uniform(0.3, 0.8), 2),
                    prec=rng.choice([32, 32, 64]), mode=rng.choice(["fast", "fast", "engine"]), tile=tile,
                    scheduler=sched)
    if kind == "forward":
        tile, sched = rng.choice([(6, 1), (6, 0), (0, 0), (5, 0)])
        nx = _log(rng, 41, 241)
        stations = max(1, min(30, int(30 * (121 / nx) ** 3), _log(rng, 2, 30)))
        return dict(kind=kind, nx=nx, nz=max(21, min(121, _log(rng, nx // 4, nx // 2 + 4))),
                    h=rng.choice([0.25, 0.5, 1.0]), stations=stations, events=_log(rng, 10, 400),
                    rays=_log(rng, 40, 12000), prec=rng.choice([64, 64, 32]), tile=tile, scheduler=sched)
    if kind == "rays":
        nx = _log(rng, 41, 161)
        return dict(kind=kind, nx=nx, nz=max(21, nx // 2), h=rng.choice([0.25, 0.5, 1.0]), tables=_log(rng, 1, 12),
                    rays=_log(rng, 50, 40000))
    if kind == "locate":
        nx = _log(rng, 41, 161)
        return dict(kind=kind, nx=nx, nz=max(21, nx // 2), h=rng.choice([0.5, 1.0]), stations=_log(rng, 6, 40),
                    events=_log(rng, 20, 600), share=round(rng.uniform(0.5, 0.95), 2))
    if kind == "lsqr":
        nx = _log(rng, 61, 121)
        return dict(kind=kind, nx=nx, nz=max(21, nx // 2), h=0.5, tables=_log(rng, 4, 20), rays=_log(rng, 500, 12000),
                    iterations=_log(rng, 4, 12))
    return dict(kind=kind, requests=_log(rng, 4, 24), prec=64)


# ---- models and tables ---------------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _solver(tile: int | None = None, scheduler: int = 0) -> EikonalCuda:
    """The solver a program keeps for its life: its settings, or the ones a context starts with."""
    s = EikonalCuda.create(0, 64)
    if tile is not None:
        for prec in (64, 32):
            L.check(L.load().ts_engine_set_tile(s.handle, prec, tile), s)
        L.check(L.load().ts_engine_set_scheduler(s.handle, scheduler), s)
    return s


@functools.lru_cache(maxsize=None)
def _server(prec: int) -> Server:
    # 32x8x4 pencils, flow scheduler, two rounds per epoch: the documented serving configuration.
    return Server(0, prec, L.MODE_FAST, tile=6, budget_bytes=60e9, rounds_per_epoch=2, scheduler=1)


def _axes(g: GridDef, h: float):
    t = lambda n: torch.arange(n, dtype=torch.float64, device=DEVICE) * h  # noqa: E731
    z = torch.from_numpy(np.ascontiguousarray(g.depth())).to(DEVICE)
    return t(g.nx)[None, None, :], t(g.ny)[None, :, None], z[:, None, None]


def _velocity(g: GridDef, h: float, rng: np.random.Generator, v0: float = 5.0, grad: float = 0.03,
              amplitude: float = 0.05) -> torch.Tensor:
    """Vp(z) times a checkerboard and two smooth bodies, all placed by rng (nz, ny, nx)."""
    x, y, z = _axes(g, h)
    cell = float(rng.uniform(6, 14)) * max(h, 0.25)
    ph = rng.uniform(0, np.pi, 3)
    v = (v0 + grad * z) * (1 + amplitude * torch.sin(math.pi * x / cell + ph[0]) *
                           torch.sin(math.pi * y / cell + ph[1]) * torch.sin(math.pi * z / cell + ph[2]))
    span = ((g.nx - 1) * h, (g.ny - 1) * h, float(g.depth()[-1]))
    for b in range(2):
        c = rng.uniform(0.2, 0.8, 3) * span
        a = rng.uniform(0.12, 0.3, 3) * span + 1e-9
        r2 = ((x - c[0]) / a[0]) ** 2 + ((y - c[1]) / a[1]) ** 2 + ((z - c[2]) / a[2]) ** 2
        v = v * (1 + (0.08 if b == 0 else -0.08) * torch.exp(-math.log(2) * r2 ** 3))
    return v


def _host(t: torch.Tensor, dtype=np.float64) -> np.ndarray:
    return np.ascontiguousarray(t.reshape(-1).cpu().numpy().astype(dtype, copy=False))


def _surface(g: GridDef, h: float, n: int, rng) -> np.ndarray:
    xy = rng.uniform(0.03, 0.97, (n, 2)) * [(g.nx - 1) * h, (g.ny - 1) * h]
    lon, lat = km_to_geo(g, xy[:, 0], xy[:, 1], h)
    return np.stack([lon, lat, np.zeros(n)], axis=1)


def _volume(g: GridDef, h: float, n: int, rng, lo: float = 0.06, hi: float = 0.8) -> np.ndarray:
    bottom = float(g.depth()[-1])
    x, y = rng.uniform(0.02, 0.98, n) * (g.nx - 1) * h, rng.uniform(0.02, 0.98, n) * (g.ny - 1) * h
    lon, lat = km_to_geo(g, x, y, h)
    return np.stack([lon, lat, rng.uniform(lo, hi, n) * bottom], axis=1)


def _analytic_tables(g: GridDef, h: float, stations: np.ndarray, vps: tuple[float, ...]) -> np.ndarray:
    """Float tables of the constant-gradient medium v0 + 0.03 z at every station and v0 of vps:
    t = acosh(1 + g²d²/(2 v v_s)) / g, on the grid's own Cartesian positions. (tables, n)"""
    lon, lat, dep = (torch.from_numpy(np.ascontiguousarray(a)).to(DEVICE) for a in (g.lon(), g.lat(), g.depth()))
    r = (EARTH_RADIUS_KM - dep)[:, None, None]
    cl, sl = torch.cos(lat * DEG2RAD)[None, :, None], torch.sin(lat * DEG2RAD)[None, :, None]
    co, so = torch.cos(lon * DEG2RAD)[None, None, :], torch.sin(lon * DEG2RAD)[None, None, :]
    out = torch.empty((len(vps), len(stations), g.nz, g.ny, g.nx), dtype=torch.float32, device=DEVICE)
    grad = 0.03
    for q, (slon, slat, sdep) in enumerate(stations):
        rs = EARTH_RADIUS_KM - sdep
        p = (rs * math.cos(slat * DEG2RAD) * math.cos(slon * DEG2RAD),
             rs * math.cos(slat * DEG2RAD) * math.sin(slon * DEG2RAD), rs * math.sin(slat * DEG2RAD))
        d2 = (r * cl * co - p[0]) ** 2 + (r * cl * so - p[1]) ** 2 + (r * sl - p[2]) ** 2
        for k, v0 in enumerate(vps):
            vs, gk = v0 + grad * v0 / vps[0] * sdep, grad * v0 / vps[0]
            v = v0 + gk * dep[:, None, None]
            out[k, q] = (torch.acosh(1 + gk * gk * d2 / (2 * v * vs)) / gk).float()
    return np.ascontiguousarray(out.reshape(len(vps) * len(stations), -1).cpu().numpy())


def _table_times(g: GridDef, tables: np.ndarray, pts: np.ndarray) -> np.ndarray:
    """Trilinear times of every table at every point (points, tables), in 64 bits."""
    fx, fy, fz = (np.clip(v, 0, n - 1) for v, n in
                  zip(g.fractional(pts[:, 0], pts[:, 1], pts[:, 2]), (g.nx, g.ny, g.nz)))
    i, j, k = (np.minimum(f.astype(np.int64), n - 2) for f, n in zip((fx, fy, fz), (g.nx, g.ny, g.nz)))
    tx, ty, tz = fx - i, fy - j, fz - k
    t = np.zeros((len(pts), len(tables)))
    for dk in (0, 1):
        for dj in (0, 1):
            for di in (0, 1):
                w = (tx if di else 1 - tx) * (ty if dj else 1 - ty) * (tz if dk else 1 - tz)
                t += w[:, None] * tables[:, ((k + dk) * g.ny + j + dj) * g.nx + i + di].T.astype(np.float64)
    return t


# ---- prepare -----------------------------------------------------------------------------------------

def _buffers(n_rays: int, nodes: float) -> tuple[np.ndarray, np.ndarray]:
    """Room for the columns and lengths of n_rays rows on grids of about `nodes` across (a row holds
    about 1.5 times that many; few rays vary more). The rows' number of non-zeros belongs to the seed,
    the buffers' size to the case: what no row reaches stays -1 and 0."""
    cap = int(n_rays * nodes * (2.2 + 30.0 / math.sqrt(n_rays)))
    return np.full(cap, -1, np.int32), np.zeros(cap, np.float32)


def _prepare_solve(case, rng):
    g = regular_grid(case["nx"], case["ny"], case["nz"], case["h"])
    s = _host(1 / _velocity(g, case["h"], rng))
    src = _volume(g, case["h"], case["fields"], rng, 0.0, 0.6)
    seeds = [point_source(g, s, *p) for p in src]
    out = np.empty((case["fields"], g.count), np.float64 if case["out"] == 64 else np.float32)
    return dict(solver=_solver(), grid=g, slowness=s, seeds=seeds, out=out)


def _prepare_tables(case, rng):
    g = regular_grid(case["nx"], case["ny"], case["nz"], case["h"])
    v = _velocity(g, case["h"], rng, 5.0, 0.04)
    slow = np.stack([_host(1 / v), _host(1.73 / v)])
    st = _surface(g, case["h"], case["stations"], rng)
    return dict(solver=_solver(), grid=g, slowness=slow, sources=np.concatenate([st, st]),
                phases=np.repeat(np.arange(2, dtype=np.int32), len(st)))


def _prepare_multi(case, rng):
    gen = torch.Generator(device=DEVICE).manual_seed(int(rng.integers(1 << 60)))
    dims = random.Random(f"{case['grids']} {case['scale']}")  # the sizes belong to the case, the models to the seed
    grids, slow, seeds = [], [], []
    for q in range(case["grids"]):
        nx, ny = (max(8, int(dims.randint(48, 192) * case["scale"])) for _ in range(2))
        nz = max(8, int(dims.randint(32, 96) * case["scale"]))
        h = dims.uniform(0.25, 1.0)
        depth = None
        if q % 2:
            steps = dims.uniform(1.02, 1.05) ** np.arange(nz - 1)
            depth = np.concatenate([[0.0], np.cumsum(steps)]) * ((nz - 1) * h / steps.sum())
            depth[-1] = (nz - 1) * h
        g = regular_grid(nx, ny, nz, h, depth)
        pert = torch.exp(0.04 * torch.randn((1, 1, *g.shape), dtype=torch.float64, device=DEVICE, generator=gen))
        pert = torch.nn.functional.avg_pool3d(torch.nn.functional.pad(pert, (1,) * 6, mode="replicate"), 3, 1)[0, 0]
        z = torch.from_numpy(np.ascontiguousarray(g.depth())).to(DEVICE)[:, None, None]
        s = _host(1 / ((5.0 + 0.03 * z) * pert))
        fx, fy, fz = rng.uniform(0.1, 0.9), rng.uniform(0.1, 0.9), rng.uniform(0.0, 0.5)
        grids.append(g)
        slow.append(s)
        seeds.append(point_source(g, s, g.min_lon + fx * (g.max_lon - g.min_lon),
                                  g.min_lat + fy * (g.max_lat - g.min_lat), fz * g.max_depth_km))
    return dict(solver=_solver(case["tile"], case["scheduler"]), grids=grids, slowness=slow, seeds=seeds,
                field_grid=list(range(len(grids))))


def _prepare_forward(case, rng):
    g = regular_grid(case["nx"], case["nx"], case["nz"], case["h"])
    inv = g.coarsened(2)
    v = _velocity(g, case["h"], rng)
    slow = np.empty((2, g.count))
    slow[0] = _host(1 / v)
    slow[1] = _host(1.73 / v)
    st = _surface(g, case["h"], case["stations"], rng)
    ev = _volume(g, case["h"], case["events"], rng)
    every = case["events"] * case["stations"] * 2
    pick = np.sort(rng.choice(every, size=min(case["rays"], every), replace=False))
    e, rest = np.divmod(pick, case["stations"] * 2)
    s, p = np.divmod(rest, 2)
    solver = _solver(case["tile"], case["scheduler"]) if case["tile"] else _solver()
    return dict(kernels=rays.RayKernels(inv, g, solver), slowness=slow, stations=st, events=ev,
                arrivals=np.stack([e, s, p], axis=1).astype(np.int32),
                buffers=_buffers(len(pick), math.hypot(case["nx"], case["nz"])))


def _ray_inputs(case, rng):
    g = regular_grid(case["nx"], case["nx"], case["nz"], case["h"])
    st = _surface(g, case["h"], case["tables"], rng)
    tables = _analytic_tables(g, case["h"], st, (float(rng.uniform(4.8, 5.6)),))
    return dict(solver=_solver(), grid=g, inv=g.coarsened(2), tables=tables, station=st,
                table_of=rng.integers(0, case["tables"], case["rays"]).astype(np.int32),
                events=_volume(g, case["h"], case["rays"], rng),
                buffers=_buffers(case["rays"], math.hypot(case["nx"], case["nz"])))


class _RowsOnDevice:
    """The rows of a ray call, left on the device (a ts_rows handle), as a program keeps them for LSQR."""

    def __init__(self, s: dict):
        lib, P = L.load(), C.POINTER
        fs, is_ = s["grid"].struct(), s["inv"].struct()
        self.handle = C.c_void_p()
        rc = lib.ts_rays_trace(s["solver"].handle, C.byref(fs), len(s["tables"]),
                               s["tables"].ctypes.data_as(P(C.c_float)), s["station"].ctypes.data_as(P(C.c_double)),
                               C.byref(is_), len(s["table_of"]), s["table_of"].ctypes.data_as(P(C.c_int32)),
                               s["events"].ctypes.data_as(P(C.c_double)), rays.step_km(s["grid"], s["inv"]),
                               C.byref(self.handle))
        L.check(rc, s["solver"])

    def __del__(self):
        if self.handle:
            L.load().ts_rows_free(self.handle)
            self.handle = None


def _prepare_lsqr(case, rng):
    s = _ray_inputs(case, rng)
    return dict(solver=s["solver"], rows=_RowsOnDevice(s), n=s["inv"].count, b=rng.normal(0, 0.1, case["rays"]),
                iterations=case["iterations"], inputs=s)


def _prepare_locate(case, rng):
    g = regular_grid(case["nx"], case["nx"], case["nz"], case["h"])
    st = _surface(g, case["h"], case["stations"], rng)
    tables = _analytic_tables(g, case["h"], st, (5.0, 5.0 / 1.73))
    truth = _volume(g, case["h"], case["events"], rng, 0.15, 0.75)
    n_ev, nt = len(truth), len(tables)
    corr = rng.normal(0, 0.05, nt)
    tt = _table_times(g, tables, truth)
    # Who was picked at which table belongs to the case (the sizes), the picks to the seed.
    take = np.random.default_rng([n_ev, nt, int(100 * case["share"])]).random((n_ev, nt)) < case["share"]
    take[:, : min(nt, 6)] = True
    gross = np.where(rng.random((n_ev, nt)) < 0.03, rng.uniform(1.0, 3.0, (n_ev, nt)), 0.0)
    obs = rng.uniform(-1, 1, (n_ev, 1)) + tt + corr + rng.normal(0, 0.03, (n_ev, nt)) + gross
    quality = rng.choice(np.array([1.0, 0.75, 0.5, 0.25]), size=(n_ev, nt), p=[0.5, 0.25, 0.15, 0.1])
    start = truth.copy()
    start[:, :2] += rng.normal(0, 3.0, (n_ev, 2)) / 111.0
    start[:, 0] = np.clip(start[:, 0], g.min_lon, g.max_lon)
    start[:, 1] = np.clip(start[:, 1], g.min_lat, g.max_lat)
    start[:, 2] = np.clip(start[:, 2] + rng.normal(0, 2.0, n_ev), 0, g.max_depth_km)
    offsets = np.concatenate([[0], np.cumsum(take.sum(axis=1))]).astype(np.int32)
    ev, tb = np.nonzero(take)
    solver = _solver()
    return dict(solver=solver, tables=_TablesOnDevice(solver, g, tables),
                args=(start, offsets, tb.astype(np.int32), obs[ev, tb], quality[ev, tb], corr[tb],
                      np.concatenate([st, st])[:, :2]))


class _TablesOnDevice:
    """Resident tables, given back with the state that holds them."""

    def __init__(self, solver, g, tables):
        self.tables = location.Tables.upload(solver, g, tables)

    def __del__(self):
        self.tables.close()


def _prepare_serve(case, rng):
    sv = _server(case["prec"])
    specs, n_rays = [], 0
    sizes = np.random.default_rng(case["requests"])  # the rays of each request belong to the case
    g121, g81, g161 = regular_grid(121, 121, 61, 0.5), regular_grid(81, 81, 41, 1.0), regular_grid(161, 161, 81, 0.5)
    v121, v81, v161 = _velocity(g121, 0.5, rng), _velocity(g81, 1.0, rng), _velocity(g161, 0.5, rng, 5.0, 0.04)
    s121 = np.stack([_host(1 / v121), _host(1.73 / v121)])
    s81 = _host(1 / v81)[None]
    s161 = np.stack([_host(1 / v161), _host(1.73 / v161)])
    mid = {k: sv.model_put(g, s) for k, g, s in (("f", g121, s121), ("c", g81, s81), ("r", g161, s161))}
    for q in range(case["requests"]):
        # 60 % one station field with 20-150 rays, 25 % resolution batches of 25 fields, 15 % relocation
        # fields with 10-40 rays: the serving load's shares, dealt in turn.
        u = (q * 0.37) % 1.0
        if u < 0.60:
            kind, g, s, h, nf, nr, ph = "f", g121, s121, 0.5, 1, int(sizes.integers(20, 151)), int(rng.integers(2))
        elif u < 0.85:
            kind, g, s, h, nf, nr, ph = "c", g81, s81, 1.0, 25, 0, 0
        else:
            kind, g, s, h, nf, nr, ph = "r", g161, s161, 0.5, 1, int(sizes.integers(10, 41)), int(rng.integers(2))
        n_rays += nr
        st = _surface(g, h, nf, rng)
        specs.append(dict(model=mid[kind], phase=ph, seed_sets=[point_source(g, s[ph], *p) for p in st], origins=st,
                          ray_field=np.zeros(nr, np.int32), ray_event=_volume(g, h, nr, rng), tables=kind == "c"))
    return dict(server=sv, specs=specs, buffers=_buffers(max(1, n_rays), math.hypot(141, 71)))


def prepare(case: dict, seed: int) -> dict:
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "rays":
        state = _ray_inputs(case, rng)
    else:
        state = dict(solve=_prepare_solve, tables=_prepare_tables, multi=_prepare_multi, forward=_prepare_forward,
                     locate=_prepare_locate, lsqr=_prepare_lsqr, serve=_prepare_serve)[kind](case, rng)
    state["case"] = case
    return state


# ---- run ---------------------------------------------------------------------------------------------

def _rows(r: rays.Rows, buffers) -> dict:
    """The rows as a program that gathers them keeps them: columns and lengths in its own arrays."""
    col, length = buffers
    col[: r.nnz] = r.col
    length[: r.nnz] = r.len
    return dict(row_ptr=r.row_ptr, col=col, len=length, tcalc_grad=r.tcalc_grad, ok=r.ok)


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "solve":
        return state["solver"].solve(state["grid"], state["slowness"], state["seeds"], state["out"],
                                     mode=MODES[case["mode"]], precision=case["prec"])
    if kind == "tables":
        with location.Tables.build(state["solver"], state["grid"], state["slowness"], state["sources"],
                                   state["phases"], precision=case["prec"]) as t:
            return t.copy()
    if kind == "multi":
        return state["solver"].solve_multi(state["grids"], state["slowness"], state["field_grid"], state["seeds"],
                                           out_dtype=np.float32, mode=MODES[case["mode"]], precision=case["prec"])
    if kind == "forward":
        return _rows(state["kernels"].compute(state["slowness"], state["stations"], state["events"],
                                              state["arrivals"], precision=case["prec"]), state["buffers"])
    if kind == "rays":
        return _rows(rays.trace_rows(state["solver"], state["grid"], state["tables"], state["station"], state["inv"],
                                     state["table_of"], state["events"]), state["buffers"])
    if kind == "locate":
        r = location.locate(state["solver"], state["tables"].tables, *state["args"])
        return dict({f: r.locations[f] for f in r.locations.dtype.names}, residuals=r.residuals)
    if kind == "lsqr":
        r = lsqr.solve_rows(state["solver"], state["rows"].handle, state["n"], state["b"], damp=0.5,
                            max_iterations=state["iterations"], atol=0.0, btol=0.0, conlim=0.0)
        return dict(x=r.solution, rnorm=r.residual_norm, iterations=r.iterations)
    sv = state["server"]
    ids = [sv.submit(**spec) for spec in state["specs"]]
    done = [sv.wait(i) for i in ids]
    col, length = state["buffers"]
    at, counts, tcg = 0, [], []
    for rows in (d.rows for d in done if d.rows is not None):
        col[at: at + rows.nnz] = rows.col
        length[at: at + rows.nnz] = rows.len
        at += rows.nnz
        counts.append(np.diff(rows.row_ptr))
        tcg.append(rows.tcalc_grad)
    out = dict(status=np.array([d.status for d in done]), tables=[d.tables for d in done if d.tables is not None])
    if counts:
        out.update(counts=np.concatenate(counts), col=col, len=length, tcalc_grad=np.concatenate(tcg))
    return out


# ---- work --------------------------------------------------------------------------------------------

UPDATE_FLOPS = 60  # one upwind update: three axis terms, the sums, the root


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "solve":
        n, f = case["nx"] * case["ny"] * case["nz"], case["fields"]
        return dict(bytes=8.0 * n + f * n * case["out"] / 8, flops=2.0 * UPDATE_FLOPS * n * f)
    if kind == "tables":
        n, f = case["nx"] * case["ny"] * case["nz"], 2 * case["stations"]
        return dict(bytes=16.0 * n + 4.0 * f * n, flops=2.0 * UPDATE_FLOPS * n * f)
    if kind == "multi":
        dims = random.Random(f"{case['grids']} {case['scale']}")
        n = 0
        for q in range(case["grids"]):
            nx, ny = (max(8, int(dims.randint(48, 192) * case["scale"])) for _ in range(2))
            n += nx * ny * max(8, int(dims.randint(32, 96) * case["scale"]))
            dims.uniform(0, 1)
            if q % 2:
                dims.uniform(0, 1)
        return dict(bytes=12.0 * n, flops=2.0 * UPDATE_FLOPS * n)
    if kind == "serve":
        u = [(q * 0.37) % 1.0 for q in range(case["requests"])]
        n = sum(121 * 121 * 61 if v < 0.6 else 25 * 81 * 81 * 41 if v < 0.85 else 161 * 161 * 81 for v in u)
        return dict(bytes=4.0 * n, flops=2.0 * UPDATE_FLOPS * n)
    nx, nz = case["nx"], case["nz"]
    n = nx * nx * nz
    # A ray: about half the grid's diagonal, two steps per node, one gather of 32 B each; about three
    # inversion nodes per step at 8 B in the row.
    steps = 0.6 * math.hypot(nx, nz)
    if kind == "forward":
        f, r = 2 * case["stations"], min(case["rays"], 2 * case["stations"] * case["events"])
        return dict(bytes=16.0 * n + 4.0 * f * n + r * steps * 56.0, flops=2.0 * UPDATE_FLOPS * n * f + 500.0 * r * steps)
    if kind == "rays":
        return dict(bytes=4.0 * case["tables"] * n + case["rays"] * steps * 56.0, flops=500.0 * case["rays"] * steps)
    if kind == "lsqr":
        nnz, cols = case["rays"] * steps * 2.0, n / 8
        return dict(bytes=case["iterations"] * (16.0 * nnz + 16.0 * (case["rays"] + cols)),
                    flops=case["iterations"] * 4.0 * nnz)
    picks = 2 * case["stations"] * case["share"]
    cand = min(8000.0, float(n)) + 25.0 ** 1.5
    return dict(bytes=4.0 * 2 * case["stations"] * n, flops=case["events"] * cand * picks * 20.0)


# ---- what the outputs are in 64 bits -------------------------------------------------------------------

def _exact_field(g: GridDef, slow: np.ndarray, seed_idx, seed_t) -> np.ndarray:
    """The sweeping scheme in plain numpy: two phases (first order, then promoted terms) of rounds of
    eight plane-ordered sweeps until a round moves nothing by more than 1e-7 s."""
    nx, ny, nz = g.nx, g.ny, g.nz
    n = g.count
    rad = EARTH_RADIUS_KM - g.depth()
    hx = np.maximum(1e-9, rad[:, None] * np.cos(g.lat() * DEG2RAD)[None, :] * g.dlon * DEG2RAD)
    hy = rad * g.dlat * DEG2RAD
    I, J, K = (a.reshape(-1) for a in np.broadcast_arrays(np.arange(nx)[None, None, :], np.arange(ny)[None, :, None],
                                                          np.arange(nz)[:, None, None]))
    PX, PY = nx + 4, ny + 4
    T = np.full((nz + 4) * PY * PX, np.inf)
    at = ((K + 2) * PY + J + 2) * PX + I + 2
    fixed = np.zeros(n, bool)
    fixed[seed_idx] = True
    T[at[seed_idx]] = seed_t
    h = [hx[K, J], hy[K], np.full(n, g.ddepth)]
    step = [1, PX, PX * PY]
    planes = []
    for d in range(8):
        p = (nx - 1 - I if d & 1 else I) + (ny - 1 - J if d & 2 else J) + (nz - 1 - K if d & 4 else K)
        p = np.where(fixed, -1, p)
        order = np.argsort(p, kind="stable")
        cut = np.searchsorted(p[order], np.arange(nx + ny + nz - 1))
        planes.append([order[a:b] for a, b in zip(cut[:-1], cut[1:])])
    planes = [[q for q in pl if len(q)] for pl in planes]

    def root(w, t, low, s2):
        with np.errstate(invalid="ignore"):
            sw, swt, swt2 = w.sum(0), (w * t).sum(0), (w * t * t).sum(0)
            disc = swt * swt - sw * (swt2 - s2)
            r = (swt + np.sqrt(np.where(disc < 0, np.nan, disc))) / sw
            return r, (disc >= 0) & ~(r < low)

    for phase in range(2):
        for _ in range(max(32, (nx + ny + nz) // 4)):
            moved = False
            for pl in planes:
                for q in pl:
                    c = at[q]
                    te, we, tn = [], [], []
                    for ax in range(3):
                        m, p = T[c - step[ax]], T[c + step[ax]]
                        side = m <= p
                        first = np.where(side, m, p)
                        second = np.where(side, T[c - 2 * step[ax]], T[c + 2 * step[ax]])
                        w1, he = 1 / (h[ax][q] * h[ax][q]), 2 * h[ax][q] / 3
                        up = np.isfinite(second) & (second <= first) & (phase == 1)
                        ok = np.isfinite(first)
                        with np.errstate(invalid="ignore"):
                            te.append(np.where(up, (4 * first - second) / 3, first))
                        we.append(np.where(ok, np.where(up, 1 / (he * he), w1), 1.0))
                        tn.append(first)
                    te, we, tn = np.array(te), np.array(we), np.array(tn)
                    order = np.argsort(te, axis=0, kind="stable")
                    te, we, tn = (np.take_along_axis(a, order, 0) for a in (te, we, tn))
                    used = np.isfinite(te).sum(0)
                    s2 = slow[q] * slow[q]
                    cand = np.full(len(q), np.inf)
                    for k in (1, 2, 3):
                        has = used >= k
                        if has.any():
                            r, good = root(we[:k], np.where(has, te[:k], 0.0), tn[:k].max(0), s2)
                            cand = np.where(has & good, r, cand)
                    cur = T[c]
                    lower = cand < cur
                    if lower.any():
                        with np.errstate(invalid="ignore"):
                            moved |= bool((~np.isfinite(cur) | (cur - cand > 1e-7))[lower].any())
                        T[c[lower]] = cand[lower]
            if not moved:
                break
    return T[at]


def _exact_tcalc(s: dict) -> np.ndarray:
    """Time and gradient of each ray's table at its event (east, north, down), in 64 bits."""
    g, ev = s["grid"], s["events"]

    def at(fx, fy, fz):
        f = [np.clip(v, 0, n - 1) for v, n in zip((fx, fy, fz), (g.nx, g.ny, g.nz))]
        i = [np.minimum(v.astype(np.int64), n - 2) for v, n in zip(f, (g.nx, g.ny, g.nz))]
        t = [v - q for v, q in zip(f, i)]
        out = np.zeros(len(ev))
        for c in range(8):
            d = (c & 1, c >> 1 & 1, c >> 2)
            w = np.prod([v if e else 1 - v for v, e in zip(t, d)], axis=0)
            out += w * s["tables"][s["table_of"], ((i[2] + d[2]) * g.ny + i[1] + d[1]) * g.nx + i[0] + d[0]]
        return out

    f = g.fractional(ev[:, 0], ev[:, 1], ev[:, 2])
    half = [[0.5 if a == b else 0.0 for b in range(3)] for a in range(3)]
    diff = [at(*(v + o for v, o in zip(f, half[a]))) - at(*(v - o for v, o in zip(f, half[a]))) for a in range(3)]
    r = EARTH_RADIUS_KM - ev[:, 2]
    return np.stack([at(*f), diff[0] / (r * np.cos(ev[:, 1] * DEG2RAD) * g.dlon * DEG2RAD),
                     diff[1] / (r * g.dlat * DEG2RAD), diff[2] / g.ddepth], axis=1)


def _exact_lsqr(s: dict) -> dict:
    """The damped bidiagonalisation's iterates (Paige and Saunders 1982), in plain numpy."""
    r = rays.trace_rows(s["inputs"]["solver"], s["inputs"]["grid"], s["inputs"]["tables"], s["inputs"]["station"],
                        s["inputs"]["inv"], s["inputs"]["table_of"], s["inputs"]["events"])  # the input matrix
    val, col = r.len.astype(np.float64), r.col
    row = np.repeat(np.arange(r.n_rows), np.diff(r.row_ptr))
    av = lambda x: np.bincount(row, val * x[col], minlength=r.n_rows)  # noqa: E731
    atv = lambda y: np.bincount(col, val * y[row], minlength=s["n"])  # noqa: E731
    damp, u = 0.5, s["b"].copy()
    beta = np.linalg.norm(u)
    u /= beta
    v = atv(u)
    alpha = np.linalg.norm(v)
    v /= alpha
    w, x, rhobar, phibar, damped2 = v.copy(), np.zeros(s["n"]), alpha, beta, 0.0
    for _ in range(s["iterations"]):
        u = av(v) - alpha * u
        beta = np.linalg.norm(u)
        u /= beta
        v = atv(u) - beta * v
        alpha = np.linalg.norm(v)
        v /= alpha
        rhobar1 = math.hypot(rhobar, damp)
        psi = damp / rhobar1 * phibar
        phibar *= rhobar / rhobar1
        rho = math.hypot(rhobar1, beta)
        theta, rhobar, phi, phibar = beta / rho * alpha, -rhobar1 / rho * alpha, rhobar1 / rho * phibar, beta / rho * phibar
        x += phi / rho * w
        w = v - theta / rho * w
        damped2 += psi * psi
    return dict(x=x, rnorm=math.sqrt(phibar * phibar + damped2), iterations=None)


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "solve" and case["fields"] * case["nx"] * case["ny"] * case["nz"] <= 130_000:
        s = prepare(case, seed)
        return np.stack([_exact_field(s["grid"], s["slowness"], *q) for q in s["seeds"]])
    if kind == "rays":
        return dict(row_ptr=None, col=None, len=None, tcalc_grad=_exact_tcalc(prepare(case, seed)), ok=None)
    if kind == "lsqr":
        return _exact_lsqr(prepare(case, seed))
    return None  # whole steps and larger fields: minutes in plain numpy
