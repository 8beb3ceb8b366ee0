"""The work that users of the flow-step library have it do, as cases that can be timed.

A case is one run of an event over an output interval, as a program built on the library
takes it: the handle with its mesh, bed and forcing is at hand, `run` loads the event's
initial fields, advances them by a number of steps through the public entry points
(`FlowB200.run`, `FlowB200.flow_step`, `ScenarioPool.run`, `FlowB200.adapt`) and fetches
the fields, as a map output does.  Initial and fetched fields lie in page-locked arrays.
A further call runs the event again (`adapt`: advances it by another interval).

Kinds of case (`kind`):
  loop   a host program's own time loop: one `flow_step` per step, dt read back each time
  run    the device-resident loop on a single-level mesh
  amr    the same on a quadtree of several levels
  adapt  a refinement pass, then steps on the new mesh
  pool   an ensemble of small scenarios: admitted, advanced together, taken out again

Scenes (`scene`): `island` (solitary wave running up a conical island, Manning friction),
`coast` (storm surge over a sloping, partly dry coast; per-cell roughness; the high ground
behind it is left out of the mesh), `lake` (a bump of water leaving through absorbing
sides), `rain` (rain on fractal terrain with a lake) and `tsunami` (deep water, a ridge).
All inputs are synthetic and follow from the seed.

`exact` restates the two-stage scheme on single-level meshes in 64-bit torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from bg_flood_b200.adapt import depth_or_slope
from bg_flood_b200.flow import FlowB200, Loop
from bg_flood_b200.mesh import boundary_segments, uniform_mesh
from bg_flood_b200.params import BndSegmentSpec, Param
from bg_flood_b200.pool import ScenarioPool

G = 9.81
DEV = "cuda" if torch.cuda.is_available() else "cpu"


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # the smallest meshes people couple to a host model: one call per step, latency counts
        _case("coupled_128", "loop", "island", 128, 128, steps=24),
        # a small ordinary run with the library's defaults (bit-exact arithmetic), ragged size
        _case("lake_400x272_default", "run", "lake", 400, 272, steps=80, fast=0),
        # a town-scale run, not square
        _case("island_848x528", "run", "island", 848, 528, steps=100),
        # the benchmark's run-up
        _case("island_1024", "run", "island", 1024, 1024, steps=100),
        # the Kurganov engine on a ragged grid
        _case("kurganov_1520x656", "run", "lake", 1520, 656, steps=80, engine=2),
        # a coastal inundation: dry land, roughness map, mesh without the high ground
        _case("coast_1584x1056", "run", "coast", 1584, 1056, steps=80),
        # rain on grid as a parameter file sets it up: rain forces double precision
        _case("rain_640x448_double", "run", "rain", 640, 448, steps=40, fast=0, double=1),
        # deep water in split precision
        _case("tsunami_768x512_split", "run", "tsunami", 768, 512, steps=120, split=1),
        # the largest grid of the benchmark: state far above L2
        _case("island_4096", "run", "island", 4096, 4096, steps=40),
        # quadtree rain on grid, levels 0-2
        _case("amr_rain_1024_l2", "amr", "rain", 1024, 1024, steps=80, levels=2),
        # a quadtree that follows the flow, default arithmetic
        _case("adapt_lake_512_l2", "adapt", "lake", 512, 512, steps=20, levels=2, fast=0),
        # an ensemble of small scenarios
        _case("pool_32_members", "pool", "mixed", 512, 256, steps=150, members=32),
    ]


def _case(name, kind, scene, nx, ny, steps, engine=1, fast=1, double=0, split=0, levels=0, members=0):
    c = dict(kind=kind, scene=scene, nx=nx, ny=ny, steps=steps, engine=engine, fast=fast, double=double, split=split,
             levels=levels, members=members)
    if name:
        c["name"] = name
    return c


def draw(rng):
    log = lambda lo, hi: math.exp(rng.uniform(math.log(lo), math.log(hi)))
    kind = rng.choice(["loop", "run", "run", "run", "run", "run", "amr", "adapt", "pool"])
    aspect = rng.uniform(0.5, 2.0)

    def size(lo, hi):  # cells, sides in whole blocks of 16
        n = log(lo, hi)
        return (16 * max(2, round(math.sqrt(n * aspect) / 16)), 16 * max(2, round(math.sqrt(n / aspect) / 16)))

    if kind == "loop":
        nx, ny = size(5e3, 2e5)
        return _case(None, kind, rng.choice(["island", "lake", "coast"]), nx, ny, rng.randrange(8, 33),
                     engine=rng.choice([1, 1, 2]), fast=rng.choice([0, 1]))
    if kind == "run":
        scene = rng.choice(["island", "island", "coast", "coast", "lake", "rain", "tsunami"])
        split = 1 if scene == "tsunami" else 0
        double = rng.choice([0, 1]) if scene == "rain" else 0
        nx, ny = size(2e4, 1.2e6 if double or split else 1.2e7)
        return _case(None, kind, scene, nx, ny, rng.randrange(20, 61), engine=rng.choice([1, 1, 1, 2]),
                     fast=0 if double else rng.choice([0, 1, 1]), double=double, split=split)
    if kind == "amr":
        nx, ny = size(4e4, 1e6)
        return _case(None, kind, rng.choice(["rain", "coast"]), nx, ny, rng.randrange(10, 61), levels=rng.choice([1, 2]),
                     engine=rng.choice([1, 1, 2]), fast=rng.choice([0, 1, 1]))
    if kind == "adapt":
        nx, ny = size(2e4, 3e5)
        return _case(None, kind, "lake", nx, ny, rng.randrange(10, 31), levels=rng.choice([1, 2]), fast=0)
    return _case(None, kind, "mixed", 16 * rng.randrange(12, 33), 16 * rng.randrange(8, 25), rng.randrange(60, 151),
                 fast=rng.choice([0, 1, 1]), members=rng.randrange(8, 41))


# ---------------------------------------------------------------- scenes

class Scene:
    """Fields of a scene as functions of the cell-centre coordinates, its parameters and
    its forcing, all from the seed."""

    def __init__(self, case, seed, scene=None, nx=None, ny=None):
        self.scene = scene or case["scene"]
        self.nx, self.ny = nx or case["nx"], ny or case["ny"]
        r = np.random.default_rng([int(seed), 17])
        site = np.random.default_rng([self.nx, self.ny, 29])  # geography of a site, the same for every event
        self.rain, self.film = None, 0.0
        p = Param(xo=0.0, yo=0.0, engine=case["engine"], aoibnd=0, fastmath=case["fast"],
                  doubleprecision=case["double"], splitprecision=case["split"])
        n = max(self.nx, self.ny)
        if self.scene == "island":
            p.dx = 51.2 / n
            p.cf, p.frictionmodel = 0.01, -1
            self.c = (r.uniform(0.45, 0.55) * self.nx * p.dx, r.uniform(0.45, 0.55) * self.ny * p.dx)
            amp, depth = r.uniform(0.025, 0.045), 0.32
            k = math.sqrt(3 * amp / (4 * depth ** 3))
            t = np.linspace(0.0, 20.0, 201)
            wl = amp / np.cosh(k * (math.sqrt(G * depth * (1 + amp / depth)) * t - 1.0 / k)) ** 2
            p.segments = [BndSegmentSpec("left", 2, list(t), list(wl))]
            self.wave = (r.uniform(0.15, 0.35) * self.nx * p.dx, 0.02)
        elif self.scene == "coast":
            p.dx = 10.0
            p.cf, p.frictionmodel = 0.02, -1
            p.mask = 14.0
            t = np.linspace(0.0, 7200.0, 241)  # (high water ends with the series)
            p.segments = [BndSegmentSpec("left", 2, list(t), list(r.uniform(0.8, 1.8) * np.sin(2 * math.pi * t / 3600.0)))]
            self.modes = _modes(site, 12, self.nx * p.dx, self.ny * p.dx)
            self.wave = (r.uniform(0.2, 0.4), r.uniform(0.5, 1.5))
        elif self.scene == "lake":
            p.dx = 2.0
            p.cf, p.frictionmodel = 0.002, 0
            p.zsinit = 0.0
            p.aoibnd = 3 if case["kind"] != "adapt" else 0
            self.c = (r.uniform(0.3, 0.7) * self.nx * p.dx, r.uniform(0.3, 0.7) * self.ny * p.dx)
            self.amp = r.uniform(0.3, 0.6)
            self.modes = _modes(r, 6, self.nx * p.dx, self.ny * p.dx)
        elif self.scene == "rain":
            p.dx = 10.0
            p.cf, p.frictionmodel = 0.035, -1
            self.modes = _modes(r, 40, self.nx * p.dx, self.ny * p.dx)
            rate = float(r.uniform(30.0, 90.0))
            self.rain = ([0.0, 3600.0, 3601.0, 1e9], [rate, rate, 0.0, 0.0])
            self.film = r.uniform(0.002, 0.006)  # water already on the ground, in the middle of an event
        else:  # tsunami
            p.dx = 500.0
            p.cf, p.frictionmodel = 0.0, 0
            self.c = (r.uniform(0.2, 0.4) * self.nx * p.dx, r.uniform(0.4, 0.6) * self.ny * p.dx)
            self.amp = r.uniform(0.3, 1.0)
        self.param = p

    def bed(self, x, y):
        p, lx, ly = self.param, self.nx * self.param.dx, self.ny * self.param.dx
        if self.scene == "island":
            d = torch.sqrt((x - self.c[0]) ** 2 + (y - self.c[1]) ** 2)
            return -0.32 + torch.clamp((3.6 - d) / 2.5, 0.0, 1.0) * 0.625
        if self.scene == "coast":  # -10 m offshore, the shore at half way, 18 m inland
            s = x / lx
            return torch.where(s < 0.5, 20.0 * (s - 0.5), 36.0 * (s - 0.5)) + 1.2 * _field(self.modes, x, y)
        if self.scene == "lake":
            return -3.0 + 0.4 * _field(self.modes, x, y)
        if self.scene == "rain":  # relief of some 100 m with a valley along the middle
            return (60.0 + 10.0 * _field(self.modes, x, y)) * (1 - 0.8 * torch.exp(-((y / ly - 0.5) / 0.08) ** 2))
        return -4000.0 + 3800.0 * torch.exp(-((x - 0.7 * lx) / (0.08 * lx)) ** 2)

    def level(self, x, y):
        """Initial water surface (dry where the bed is above it)."""
        p, lx = self.param, self.nx * self.param.dx
        if self.scene == "island":
            return self.wave[1] * torch.exp(-((x - self.wave[0]) / 2.0) ** 2)
        if self.scene == "coast":
            return self.wave[1] * torch.exp(-((x - self.wave[0] * lx) / (0.05 * lx)) ** 2)
        if self.scene == "lake":
            return self.amp * torch.exp(-((x - self.c[0]) ** 2 + (y - self.c[1]) ** 2) / (2 * 40.0 ** 2))
        if self.scene == "rain":
            return torch.full_like(x, 12.0)
        return self.amp * torch.exp(-((x - self.c[0]) ** 2 + (y - self.c[1]) ** 2) / (2 * (0.05 * lx) ** 2))

    def roughness(self, x, y):
        return 0.02 + 0.03 * torch.sigmoid(_field(self.modes, x, y)) if self.scene == "coast" else None

    # fields on the library's tiles (nblk, 18, 18) from block origins and cell sizes
    def tiles(self, bxo, byo, dxl):
        t = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=DEV)
        i = torch.arange(-1, 17, device=DEV, dtype=torch.float64)
        d = t(dxl)[:, None, None]
        x = t(bxo)[:, None, None] + i[None, None, :] * d + 0 * i[None, :, None]
        y = t(byo)[:, None, None] + i[None, :, None] * d + 0 * i[None, None, :]
        # coordinates of the cell centres (a block's origin is its first cell's)
        x, y = x + 0.5 * self.param.dx, y + 0.5 * self.param.dx
        zb = self.bed(x, y).float().double()
        h = torch.clamp(self.level(x, y) - zb, min=self.film).float().double()
        cf = self.roughness(x, y)
        return zb, h, None if cf is None else cf.float().double()

    def mesh(self):
        p = self.param
        present = None
        if self.scene == "coast":
            whole = uniform_mesh(self.nx, self.ny, p.dx, doubleprecision=bool(p.doubleprecision))
            zb, _, _ = self.tiles(whole.xo, whole.yo, np.full(whole.nblk, p.dx))
            present = (zb[:, 1:17, 1:17] < p.mask).flatten(1).any(1).cpu().numpy().reshape(whole.nby, whole.nbx)
        return uniform_mesh(self.nx, self.ny, p.dx, present=present, doubleprecision=bool(p.doubleprecision))


def _modes(r, n, lx, ly):
    """Random waves, amplitude falling with the wave number (longest: the domain)."""
    k = np.exp(r.uniform(0.0, math.log(24.0), n))
    a = r.uniform(0, 2 * math.pi, n)
    return [(2 * math.pi * kk * math.cos(t) / max(lx, ly), 2 * math.pi * kk * math.sin(t) / max(lx, ly), ph, 1.0 / kk ** 0.8)
            for kk, t, ph in zip(k, a, r.uniform(0, 2 * math.pi, n))]


def _field(modes, x, y):
    z = torch.zeros_like(x)
    for kx, ky, ph, a in modes:
        z += a * torch.cos(kx * x + ky * y + ph)
    return z


# ---------------------------------------------------------------- handles

def _handle(scene, mem=None, adaptive=False):
    """(handle, mesh) of a scene, loaded through the library's calls."""
    p, mesh = scene.param, scene.mesh()
    mem = mesh.nblk if mem is None else max(mem, mesh.nblk)
    f = FlowB200(p, mem)
    zb, h, cf = scene.tiles(mesh.xo, mesh.yo, np.full(mesh.nblk, p.dx))

    def host(a):
        out = np.zeros((mem, 18, 18), f.dtype)
        out[: mesh.nblk] = a.to(torch.float64 if f.dtype == np.float64 else torch.float32).cpu().numpy()
        return out

    f.set_blocks(mesh.active, mesh.level, mesh.nbr, mesh.xo, mesh.yo)
    f.set_bed(host(zb), cf=None if cf is None else host(cf))
    for typ, times, levels, sides in boundary_segments(mesh, p.segments, p.aoibnd, 0.0, 0.0):
        f.add_segment(typ, times, levels, sides)
    if scene.rain is not None:
        f.set_rain(*scene.rain)
    z = np.zeros((mem, 18, 18), f.dtype)
    f.set_state(host(h), z, z)
    if adaptive:
        gx, gy = torch.meshgrid((torch.arange(scene.nx, device=DEV, dtype=torch.float64) + 0.5) * p.dx,
                                (torch.arange(scene.ny, device=DEV, dtype=torch.float64) + 0.5) * p.dx, indexing="xy")
        f.set_bathy(0.5 * p.dx, 0.5 * p.dx, p.dx, scene.bed(gx, gy).float().cpu().numpy())
    return f, mesh


def _fields(f, n):
    """Page-locked arrays for fields, kept by the program."""
    dt = torch.float64 if f.dtype == np.float64 else torch.float32
    pin = torch.cuda.is_available()
    return [torch.zeros((f.nblkmem, 18, 18), dtype=dt, pin_memory=pin).numpy() for _ in range(n)]


def _start(f):
    loop = Loop(nextoutputtime=1e30)
    f.init_dt(loop)
    return loop


def _criterion(case):
    # rain: where water stands; lake: the passing wave; coast: deeper water and steep surfaces
    return depth_or_slope(0.05, 1e9) if case["scene"] == "rain" else \
        depth_or_slope(1e9, 2e-3) if case["scene"] == "lake" else depth_or_slope(2.0, 1e-3)


def prepare(case, seed):
    if case["kind"] == "pool":
        members = []
        for s in _members(case, seed):
            f, mesh = _handle(s)
            members.append((f, mesh.nblk, _start(f)))
        pool = ScenarioPool(members[0][0].param, sum(n for _, n, _ in members), len(members))
        return dict(case=case, pool=pool, members=members)
    s = Scene(case, seed)
    if case["kind"] in ("amr", "adapt"):
        n0 = (case["nx"] // 16) * (case["ny"] // 16)
        s.param.initlevel, s.param.minlevel, s.param.maxlevel = 0, 0, case["levels"]
        f, _ = _handle(s, mem=n0 * (4 ** case["levels"] + 4), adaptive=True)
        f.adapt(_criterion(case), maxiteration=case["levels"] + 1, allow_coarsen=True)
    else:
        f, _ = _handle(s)
    first, out = _fields(f, 3), _fields(f, 4)
    for a, b in zip(first, f.get_state(out=out)[1:]):
        a[:] = b
    return dict(case=case, f=f, loop=_start(f), first=first, out=out)


def _members(case, seed):
    """Scenes of an ensemble: block counts log-uniform up to the case's size."""
    r, sizes = np.random.default_rng([int(seed), 23]), np.random.default_rng(23)
    got = []
    for k in range(case["members"]):
        u = math.exp(sizes.uniform(math.log(0.28), 0.0))
        nx, ny = (16 * max(2, round(u * v / 16)) for v in (case["nx"], case["ny"]))
        got.append(Scene(case, int(r.integers(1 << 30)), scene=("rain", "coast", "rain", "lake")[k % 4], nx=nx, ny=ny))
    return got


def run(state):
    case = state["case"]
    if case["kind"] == "pool":
        pool, members = state["pool"], state["members"]
        slots = [pool.admit(f, loop, 1e30, maxsteps=case["steps"]) for f, _, loop in members]
        pool.run(case["steps"])
        return {"h": [r[1] for r in pool.finish(slots, [n for _, n, _ in members])]}
    f, loop = state["f"], state["loop"]
    got = {}
    if case["kind"] == "adapt":
        f.adapt(_criterion(case), maxiteration=case["levels"] + 1, allow_coarsen=True)
    else:
        f.set_state(*state["first"])
        loop = Loop(nextoutputtime=loop.nextoutputtime, dtmax=loop.dtmax)
    if case["kind"] == "loop":
        dts = np.empty(case["steps"])
        for k in range(case["steps"]):
            dts[k] = f.flow_step(loop)
            loop.totaltime += loop.dt
        got["dts"] = dts
    else:
        f.run(loop, 1e30, maxsteps=case["steps"])
    zs, h, u, v = f.get_state(out=state["out"])
    got.update(zs=zs, h=h, u=u, v=v, dt=loop.dt, time=loop.totaltime)
    if case["kind"] == "adapt":
        active, level, nbr, xo, yo = f.get_blocks()
        tables = np.full((f.nblkmem, 10), -1, np.int32)  # of the active blocks, in their order
        tables[: len(active)] = np.column_stack([active, level[active], nbr[active]])
        got["tables"] = tables
    return got


# ---------------------------------------------------------------- work and tolerance

def _cells(case):
    n = case["nx"] * case["ny"]
    if case["kind"] == "pool":
        return int(0.35 * n * case["members"])
    if case["kind"] in ("amr", "adapt"):
        return int(n * 4 ** case["levels"] * 0.4)
    return int(0.8 * n) if case["scene"] == "coast" else n


def work(case):
    # a step reads h, u, v and the bed and writes h, u, v; a pass also reads the initial
    # fields and writes the fetched ones.  About 700 operations per cell and step: two
    # stages of eight limited slopes, two reconstructed Riemann problems and an advance.
    size = 8 if case["double"] else 4
    n, k = _cells(case), case["steps"]
    io = 4 if case["kind"] == "pool" else 7
    return {"bytes": float(n) * (k * 7 * size + io * size), "flops": 700.0 * n * k}


def tolerance(case):
    # four times the largest difference between the two arithmetic builds on these scenes;
    # velocities that start from rest (a tsunami's, the alongshore one of a coast) are small
    # against the rounding of the depth under them
    if case["double"]:
        return {"rel": 1e-12, "max": 1e-9}
    if case["kind"] == "adapt":
        return {"rel": 1e-6, "max": 1e-4, "differ": 0.0}  # (default arithmetic: the mesh is the same)
    if case["scene"] == "tsunami":
        return {"rel": 6e-3, "max": 8e-2}
    if case["scene"] in ("coast", "mixed"):
        return {"rel": 3e-3, "max": 4e-2}
    return {"rel": 7e-4, "max": 3e-2}


# ---------------------------------------------------------------- 64-bit restatement

def exact(case, seed):
    if case["levels"]:
        return None  # the cross-level halo rules are not restated here
    if case["kind"] == "pool":
        scenes = _members(case, seed)
        h, _, _, _, _, _, n = _Exact(scenes).advance(case["steps"])
        got, b = [], 0
        for k in n:
            got.append(h[b: b + k].cpu().numpy())
            b += k
        return {"h": got}
    s = Scene(case, seed)
    e = _Exact([s])
    h, u, v, zb, dts, time, _ = e.advance(case["steps"])

    def tile(a):
        out = np.zeros((a.shape[0], 18, 18))
        out[:, 1:17, 1:17] = a.cpu().numpy()
        return out

    got = {"zs": tile(zb + h), "h": tile(h), "u": tile(u), "v": tile(v), "dt": dts[-1], "time": time}
    if case["kind"] == "loop":
        got["dts"] = np.array(dts)
    return got


class _Exact:
    """The two-stage step on single-level block meshes, one or several scenarios at
    once (blocks one after the other, a dt for each scenario)."""

    def __init__(self, scenes):
        self.scenes, self.p = scenes, scenes[0].param
        meshes = [s.mesh() for s in scenes]
        self.n = [m.nblk for m in meshes]
        off = np.concatenate([[0], np.cumsum(self.n)])
        nbr = np.concatenate([m.nbr + o for m, o in zip(meshes, off)])
        ids = np.arange(len(nbr))
        T = lambda a, dt=torch.float64: torch.as_tensor(np.asarray(a), device=DEV, dtype=dt)
        self.sc = T(np.repeat(np.arange(len(scenes)), self.n), torch.int64)
        zb, h, cf = zip(*(s.tiles(m.xo, m.yo, np.full(m.nblk, s.param.dx)) for s, m in zip(scenes, meshes)))
        inner = lambda a: a[:, 1:17, 1:17].contiguous()
        self.zb, self.h = (torch.cat([inner(x) for x in a]) for a in (zb, h))
        # the roughness and the step's other parameters, by block where they differ
        blk = lambda vals: T([vals[i] for i in range(len(scenes))])[self.sc][:, None, None]
        P = [s.param for s in scenes]
        f32 = (lambda v: float(np.float32(v))) if not self.p.doubleprecision else float
        self.cf = torch.cat([inner(c) if c is not None else torch.full_like(inner(z), f32(q.cf))
                             for c, z, q in zip(cf, zb, P)])
        self.delta = blk([f32(q.dx) for q in P])
        self.model = blk([float(q.frictionmodel) for q in P])
        self.eps = f32(self.p.eps)
        self.theta, self.cfl, self.g = f32(self.p.theta), f32(self.p.CFL), f32(G)
        # tile source of each cell of the 20x20 tile: a neighbour's cell, or the block's own
        # edge cell at the end of the mesh
        src = np.zeros((len(nbr), 20, 20), np.int64)
        y, x = np.mgrid[-2:18, -2:18]
        for cond, side, dx, dy in (((x < 0), 0, 16, 0), ((x > 15), 2, -16, 0), ((y < 0), 4, 0, 16), ((y > 15), 6, 0, -16)):
            nb = nbr[:, side]
            own = (nb == ids)[:, None]
            yy, xx = y[cond], x[cond]
            cx, cy = np.clip(xx, 0, 15), np.clip(yy, 0, 15)
            sx, sy = np.clip(xx + dx, 0, 15), np.clip(yy + dy, 0, 15)
            src[:, cond] = np.where(own, ids[:, None] * 256 + cy * 16 + cx, nb[:, None] * 256 + sy * 16 + sx)
        mid = (x >= 0) & (x < 16) & (y >= 0) & (y < 16)
        src[:, mid] = ids[:, None] * 256 + (y[mid] * 16 + x[mid])
        self.src = T(src, torch.int64)
        self.zt = self.tile(self.zb)
        self.dzx, self.dzy = self.grad_x(self.zt), self.grad_y(self.zt)
        # segments: type and series of each block side (left, right, top, bottom)
        self.segs, self.side = [], np.full((len(nbr), 4), -1)
        for s, m, o, q in zip(scenes, meshes, off, P):
            for typ, t, w, sides in boundary_segments(m, q.segments, q.aoibnd, 0.0, 0.0):
                for k in range(4):
                    self.side[np.asarray(sides[k], np.int64) + o, k] = len(self.segs)
                self.segs.append((typ, np.asarray(t), np.asarray(w), q.zsinit))
        self.qmean = torch.zeros((len(nbr), 4, 16), device=DEV, dtype=torch.float64)

    def tile(self, a):
        return a.reshape(-1)[self.src]

    def minmod(self, s0, s1, s2):
        d1, d2, d3 = self.theta * (s1 - s0), (s2 - s0) / 2, self.theta * (s2 - s1)
        up = torch.minimum(torch.minimum(d1, d2), d3)
        dn = torch.maximum(torch.maximum(d1, d2), d3)
        z = torch.zeros_like(d1)
        return torch.where((s0 < s1) & (s1 < s2), up, torch.where((s0 > s1) & (s1 > s2), dn, z))

    def grad_x(self, t):  # x = -1..16, rows 0..15
        r = t[:, 2:18]
        return self.minmod(r[:, :, 0:18], r[:, :, 1:19], r[:, :, 2:20]) / self.delta

    def grad_y(self, t):  # y = -1..16, columns 0..15
        r = t[:, :, 2:18]
        return self.minmod(r[:, 0:18], r[:, 1:19], r[:, 2:20]) / self.delta

    def wetslope(self, zs, h, zsm, zsp, dzs, dh, dzb):
        mz, pz = zs - h - self.delta / 2 * (dzs - dh), zs - h + self.delta / 2 * (dzs - dh)
        return torch.where((dzs ** 2 > dzb ** 2) & ((mz > zsm) | (pz > zsp)), dh + dzb, dzs)

    def face(self, ci, cn, gi, gn, zbi, zbn):
        """Fluxes of the faces between cells n and i: state h, zs, un, ut and gradients."""
        (hi, zsi, ui, ti), (hn, zsn, un, tn) = ci, cn
        (dhi, dzi, dui, dti), (dhn, dzn, dun, dtn) = gi, gn
        dx, ga, g = self.delta / 2, self.g / 2, self.g
        eps = self.eps + (2.0 ** -52 if self.p.doubleprecision else 2.0 ** -23)
        zero = torch.zeros_like(hi)
        wet = (hi > eps) | (hn > eps)
        if self.p.engine == 2:
            zi, zn = zsi - hi, zsn - hn
            zl, zr = zi - dx * (dzi - dhi), zn + dx * (dzn - dhn)
            zlr = torch.maximum(zl, zr)
            hl, up = hi - dx * dhi, ui - dx * dui
            hr, um = hn + dx * dhn, un + dx * dun
            hp, hm = torch.clamp(hl + zl - zlr, min=0), torch.clamp(hr + zr - zlr, min=0)
            cp, cm = torch.sqrt(g * hp), torch.sqrt(g * hm)
            ap = torch.clamp(torch.maximum(up + cp, um + cm), min=0)
            am = torch.clamp(torch.minimum(up - cp, um - cm), max=0)
            a = torch.maximum(ap, -am)
            qm, qp = hm * um, hp * up
            fh = torch.where(a > 0, (ap * qm - am * qp + ap * am * (hp - hm)) / (ap - am), zero)
            fu = torch.where(a > 0, (ap * (qm * um + ga * hm ** 2) - am * (qp * up + ga * hp ** 2) + ap * am * (qp - qm)) /
                             (ap - am), zero)
            ft = torch.where(fh > 0, tn + dx * dtn, ti - dx * dti) * fh
            sl = ga * (hp ** 2 - hl ** 2 + (hl + hi) * (zi - zl))
            sr = ga * (hm ** 2 - hr ** 2 + (hr + hn) * (zn - zr))
        else:
            hr, hl = hi - dx * dhi, hn + dx * dhn
            er, el = zsi - dx * dzi, zsn + dx * dzn
            zr, zl = er - hr, el - hl
            z = torch.minimum(torch.maximum(zr, zl), torch.minimum(el, er))
            hp = torch.clamp(torch.minimum(er - z, hr), min=0)
            hm = torch.clamp(torch.minimum(el - z, hl), min=0)
            fr = torch.where(hi > eps, (1 + dx * dhi / hi) * dx, dx + zero)
            fl = torch.where(hn > eps, (1 - dx * dhn / hn) * dx, dx + zero)
            up, vr, um, vl = ui - fr * dui, ti - fr * dti, un + fl * dun, tn + fl * dtn
            cm, cp = torch.sqrt(g * hm), torch.sqrt(g * hp)
            us, cs = (um + up) / 2 + cm - cp, (cm + cp) / 2 + (um - up) / 4
            SL = torch.where(hm == 0, up - 2 * cp, torch.minimum(um - cm, us - cs))
            SR = torch.where(hp == 0, um + 2 * cm, torch.maximum(up + cp, us + cs))
            fhm, fum = um * hm, hm * (um ** 2 + g * hm / 2)
            fhp, fup = up * hp, hp * (up ** 2 + g * hp / 2)
            fh = torch.where(SL >= 0, fhm, torch.where(SR <= 0, fhp, (SR * fhm - SL * fhp + SL * SR * (hp - hm)) / (SR - SL)))
            fu = torch.where(SL >= 0, fum, torch.where(SR <= 0, fup, (SR * fum - SL * fup + SL * SR * (fhp - fhm)) / (SR - SL)))
            a = torch.maximum(SL.abs(), SR.abs())
            ft = torch.where(fh > 0, vl, vr) * fh
            sl, sr = ga * (hi + hp) * (zbi - z), ga * (hm + hn) * (zbn - z)
        huge = 2.0 ** 52 if self.p.doubleprecision else 2.0 ** 23
        dt = torch.where(a > 1.0 / huge, self.cfl * self.delta / a, huge + zero)
        out = [torch.where(wet, q, zero) for q in (fh, fu - sl, fu - sr, ft)]
        return out, torch.where(wet, dt, huge + zero), wet

    def fluxes(self, h, u, v):
        ht, ut, vt = self.tile(h), self.tile(u), self.tile(v)
        zt = self.zt + ht
        gx = [self.grad_x(t) for t in (ht, zt, ut, vt)]
        gy = [self.grad_y(t) for t in (ht, zt, ut, vt)]
        if self.p.engine == 1:
            c = (slice(None), slice(2, 18), slice(1, 19))
            gx[1] = self.wetslope(zt[c], ht[c], zt[:, 2:18, 0:18], zt[:, 2:18, 2:20], gx[1], gx[0], self.dzx)
            c = (slice(None), slice(1, 19), slice(2, 18))
            up = zt[:, 2:20, 2:18].clone()
            up[:, 1:17] = zt[:, 1:17, 2:18]  # interior rows compare both values with the lower neighbour
            gy[1] = self.wetslope(zt[c], ht[c], zt[:, 0:18, 2:18], up, gy[1], gy[0], self.dzy)
        X = lambda a, k: a[:, 2:18, 2 + k:19 + k]
        Y = lambda a, k: a[:, 2 + k:19 + k, 2:18]
        fx, dx, wx = self.face([X(a, 0) for a in (ht, zt, ut, vt)], [X(a, -1) for a in (ht, zt, ut, vt)],
                               [g[:, :, 1:18] for g in gx], [g[:, :, 0:17] for g in gx], X(self.zt, 0), X(self.zt, -1))
        gq = [gy[0], gy[1], gy[3], gy[2]]
        fy, dy, wy = self.face([Y(a, 0) for a in (ht, zt, vt, ut)], [Y(a, -1) for a in (ht, zt, vt, ut)],
                               [g[:, 1:18] for g in gq], [g[:, 0:17] for g in gq], Y(self.zt, 0), Y(self.zt, -1))
        dx, dy, wy = dx[:, :, :16], dy[:, :16], wy[:, :16]
        return fx, fy, torch.where(wy, torch.minimum(dx, dy), dy)

    def boundaries(self, fx, fy, hn, un, vn, time):
        ht, ut, vt = self.tile(hn), self.tile(un), self.tile(vn)
        for k, (typ, ts, wl, zsinit) in enumerate(self.segs):
            if typ == 1:
                continue
            lev = 0.0 if math.isnan(zsinit) else zsinit
            for side in range(4):
                b = np.flatnonzero(self.side[:, side] == k)
                if not len(b):
                    continue
                b = torch.as_tensor(b, device=DEV)
                t = float(time[int(self.sc[b[0]])])
                if len(ts):
                    i = 1
                    while i < len(ts) - 1 and ts[i] < t:
                        i += 1
                    lev = wl[i - 1] + (t - ts[i - 1]) / (ts[i] - ts[i - 1]) * (wl[i] - wl[i - 1])
                F, low = (fx, side == 0) if side < 2 else (fy, side == 3)
                sign = -1.0 if low else 1.0
                f0, f1 = (0, 1) if low else (16, 15)  # the boundary face and the next one inside
                cell = (lambda a, c: a[b, 2:18, 2 + c]) if side < 2 else (lambda a, c: a[b, 2 + c, 2:18])
                fidx = (lambda c: (b, slice(None), c)) if side < 2 else (lambda c: (b, c, slice(None)))
                zi, zin = cell(self.zt + ht, f0), cell(self.zt + ht, f1)
                hf, hin = cell(ht, f0), cell(ht, f1)
                uin = cell(ut if side < 2 else vt, f1)
                bnd = float(np.float32(np.float32(lev)))
                f = F[0][fidx(f0)].clone()
                gq = F[1][fidx(f0)] if low else F[2][fidx(f0)]
                s = F[2][fidx(f1)] if low else F[1][fidx(f1)]
                zero = torch.zeros_like(f)
                open_ = (hf > self.eps) | (bnd > zi) if typ != 0 else torch.zeros_like(f, dtype=torch.bool)
                if typ == 3:
                    qm = self.qmean[b, side]
                    qm = torch.where(hf < 0.01, zero, 0.0 * f + qm)
                    zn, hh = torch.clamp(zi - hf, min=bnd), torch.clamp(hf, min=1e-4)
                    new = sign * torch.sqrt(self.g / hh) * (zi - zn) * hh + qm
                    self.qmean[b, side] = torch.where(open_, qm, zero)
                else:
                    zbi = zin - hin
                    new = (sign * 2 * (torch.sqrt(self.g * torch.clamp(hin, min=0)) -
                                       torch.sqrt(self.g * torch.clamp(bnd - zbi, min=0))) + uin) * hin
                F[0][fidx(f0)] = torch.where(open_, new, zero)
                (F[2] if low else F[1])[fidx(f1)] = torch.where(open_, s, gq)

    def divergence(self, fx, fy):
        d = 1.0 / self.delta
        dh = -(fx[0][:, :, 1:] - fx[0][:, :, :-1] + fy[0][:, 1:] - fy[0][:, :-1]) * d
        du = (fx[1][:, :, :-1] + fy[3][:, :-1] - fx[2][:, :, 1:] - fy[3][:, 1:]) * d
        dv = (fy[1][:, :-1] + fx[3][:, :, :-1] - fy[2][:, 1:] - fx[3][:, :, 1:]) * d
        return dh, du, dv

    def ahead(self, dt, h, u, v, dh, du, dv):
        e = torch.where(dh >= 0, dt + 0 * h, torch.minimum(dt + 0 * h, torch.clamp(h, min=self.eps) / dh.abs()))
        ho = h + e * dh
        wet = ho > self.eps
        q = torch.where(wet, ho, torch.ones_like(ho))
        z = torch.zeros_like(h)
        return ho, torch.where(wet, (h * u + e * du) / q, z), torch.where(wet, (h * v + e * dv) / q, z)

    def advance(self, steps):
        ns = len(self.scenes)
        h, z = self.h, torch.zeros_like(self.h)
        u, v = z, z.clone()
        low = lambda c: torch.full((ns,), 2.0 ** (52 if self.p.doubleprecision else 23), device=DEV,
                                   dtype=torch.float64).scatter_reduce(0, self.sc, c.flatten(1).amin(1), "amin")
        dmin = low(self.delta / torch.sqrt(self.g * torch.clamp(h, min=self.eps)))
        d0 = torch.tensor([s.param.dx for s in self.scenes], device=DEV, dtype=torch.float64)
        dtmax = torch.minimum(dmin, 1.5 * d0 / math.sqrt(G * 10.0))
        dt, time, dts = torch.zeros_like(dtmax), torch.zeros_like(dtmax), []
        for _ in range(steps):
            fx, fy, cdt = self.fluxes(h, u, v)
            self.boundaries(fx, fy, h, u, v, (time + dt / 2).tolist())
            D = self.divergence(fx, fy)
            dt = torch.minimum(low(cdt), 1.5 * dtmax)
            bdt = dt[self.sc][:, None, None]
            hs, us, vs = self.ahead(bdt / 2, h, u, v, *D)
            fx, fy, _ = self.fluxes(hs, us, vs)
            self.boundaries(fx, fy, h, u, v, (time + dt).tolist())
            h, u, v = self.ahead(bdt, h, u, v, *self.divergence(fx, fy))
            w = h > self.eps
            q = torch.where(w, h, torch.ones_like(h))
            cf = torch.where(self.model == -1, self.g * self.cf ** 2 / q ** (1.0 / 3.0), self.cf)
            fac = torch.where(w, 1 + cf * torch.sqrt(u ** 2 + v ** 2) / q * bdt, torch.ones_like(h))
            u, v = u / fac, v / fac
            if any(s.rain is not None for s in self.scenes):
                rate = [0.0 if s.rain is None else float(np.interp(t, *s.rain)) for s, t in zip(self.scenes, time.tolist())]
                r = torch.tensor(rate, device=DEV, dtype=torch.float64)[self.sc][:, None, None] / 3.6e6 * bdt
                k = torch.where(w, h / torch.where(w, h + r, torch.ones_like(h)), torch.ones_like(h))
                h, u, v = h + r, u * k, v * k
            dtmax = dt
            time = time + dt
            dts.append(float(dt[0]))
        return h, u, v, self.zb, dts, float(time[0]), self.n
