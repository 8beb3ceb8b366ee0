"""The fast build's results as bits.  Its kernels share faces between blocks, pairs and
single lanes; a face has to come out the same wherever it is formed, and a new way to split
the work must not change a result.  The digests are those of the first pair kernels (two
adjacent rows per thread, every face from the two cells' gradients), recorded on B200:
rounded products and sums, one reciprocal per star region, upwind fluxes taken as they are.

Signed zeros count as equal; everything else must be the same bits."""
import hashlib
import os

import numpy as np
import pytest

import cases
from runners import interior, make_gpu, make_gpu_amr

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(__file__), "golden")


def _set(case, **kw):
    for k, v in kw.items():
        setattr(case.param, k, v)
    case.param.fastmath = 1
    return case


def _chute(engine, **kw):
    """A thin sheet of water running down a slope of 1 : 4 into a pool: faces above the
    critical speed (Froude number 2 to 4), shocks at the foot, wetting and drying."""
    c = cases.dam_break(64, engine)
    x = (np.arange(64) + 0.5) * c.dx
    c.zb = (c.zb * 0.2 + np.maximum(24.0 - x, 0.0)[None, :] * 0.25).astype(np.float32)
    c.h = np.where(x[None, :] < 4.0, 0.5, np.maximum(0.3 - c.zb, 0.0)).astype(np.float32)
    c.u = np.where(c.h > 0, c.u + np.where(x < 24.0, 2.0, 0.0)[None, :], 0.0).astype(np.float32)
    c.v = np.where(c.h > 0, c.v, 0.0).astype(np.float32)
    return _set(c, cf=0.02, frictionmodel=-1, **kw)


def _island(n, engine, **kw):
    """The conical island with the wave already in the basin, so that all of it moves."""
    c = cases.conical_island(n, engine)
    x = (np.arange(n) + 0.5) * c.dx
    c.h = np.where(c.h > 0, np.maximum(0.03 * np.exp(-((x - 7.0) / 2.0) ** 2)[None, :] - c.zb, 0.0), 0.0).astype(np.float32)
    return _set(c, **kw)


def _amr(name, mk, rain=None, **kw):
    g = np.load(os.path.join(GOLDEN, f"{name}.npz"))
    case = _set(mk(), **kw)
    f, loop = make_gpu_amr(case, (g["level"], g["nbr"], g["xo"], g["yo"]))
    if rain:
        f.set_rain(*rain)
    return f, loop


def _reg(case):
    f, _, loop = make_gpu(case)
    return f, loop


def _sources(model, size):
    """A river on a few cells and a rain map over the whole of a square domain."""
    f, loop = model
    f.add_river(0.4 * size, 0.45 * size, 0.5 * size, 0.6 * size, [0.0, 1.0, 1e6], [0.3, 2.0, 2.0])
    yy, xx = np.mgrid[0:5, 0:5]
    f.set_rain_map(0.0, 0.0, size / 4, size / 4, 0.0, 5.0, np.stack([50.0 + 400 * (xx == k) + 7 * yy for k in range(5)]))
    return f, loop


RUNS = {
    "gauss_e1_absorbing": (lambda: _reg(_set(cases.gauss(64, 1, 3))), 40),
    "gauss_e2_absorbing": (lambda: _reg(_set(cases.gauss(64, 2, 3))), 40),
    "dam_e1": (lambda: _reg(_set(cases.dam_break(64, 1), lat=45.0)), 60),
    "dam_e2": (lambda: _reg(_set(cases.dam_break(64, 2), lat=-30.0)), 60),
    "dam_e1_mass": (lambda: _reg(_set(cases.dam_break(48, 1), ForceMassConserve=1)), 40),
    "dam_e1_smart": (lambda: _reg(_set(cases.dam_break(48, 1), cf=0.01, frictionmodel=1)), 40),
    "chute_e1": (lambda: _reg(_chute(1)), 80),
    "chute_e2": (lambda: _reg(_chute(2)), 80),
    "island_e1": (lambda: _reg(_island(96, 1)), 80),
    "island_e2": (lambda: _reg(_island(96, 2)), 80),
    "rain_e1": (lambda: _reg(_set(cases.rain_on_terrain(64, 1))), 60),
    "dam_e1_sources": (lambda: _sources(_reg(_set(cases.dam_break(64, 1), cf=0.03, frictionmodel=-1)), 32.0), 60),
    "amr_dam_e1_sources": (lambda: _sources(_amr("amrdam64_e1_l2", lambda: cases.amr_dambreak(64, 1, 2)), 32.0), 60),
    "tsunami_split": (lambda: _reg(_set(cases.ensemble_member(3, 2024, 64, 512), splitprecision=1)), 40),
    "chute_e1_split": (lambda: _reg(_chute(1, splitprecision=1)), 80),
    "chute_e2_split": (lambda: _reg(_chute(2, splitprecision=1)), 60),
    "island_e1_split": (lambda: _reg(_island(64, 1, splitprecision=1)), 40),
    "rain_e1_split": (lambda: _reg(_set(cases.rain_on_terrain(64, 1), splitprecision=1)), 40),
    "amr_dam_e1_l3": (lambda: _amr("amrdam64_e1_l3", lambda: cases.amr_dambreak(64, 1, 3)), 60),
    "amr_dam_e1_l2_rain": (lambda: _amr("amrdam64_e1_l2", lambda: cases.amr_dambreak(64, 1, 2),
                                        ([0.0, 1e9], [80.0, 80.0]), cf=0.03, frictionmodel=-1, lat=45.0), 60),
    "amr_dam_e2_l2_smart": (lambda: _amr("amrdam64_e2_l2", lambda: cases.amr_dambreak(64, 2, 2), cf=0.01,
                                         frictionmodel=1, lat=45.0), 60),
    "amr_hump_e2_l2": (lambda: _amr("amrhump64_e2_l2", lambda: cases.amr_hump(64, 2, 2, 0.3)), 40),
}


def result(name):
    mk, nsteps = RUNS[name]
    f, loop = mk()
    for _ in range(nsteps):
        loop.totaltime += f.flow_step(loop)
    _, h, u, v = f.get_state()
    return loop.totaltime, [np.ascontiguousarray(interior(a)) + 0 for a in (h, u, v)]


def digest(name):
    t, fields = result(name)
    d = hashlib.sha1(np.float64(t).tobytes())
    for a in fields:
        d.update(a.tobytes())
    return d.hexdigest()[:16]


DIGESTS = {
    "amr_dam_e1_sources": "5a9ce8073db50000",
    "dam_e1_sources": "5d9c0eaf2f43f3c8",
    "gauss_e1_absorbing": "94cfea69c87b4ad6",
    "gauss_e2_absorbing": "886228ac31590571",
    "dam_e1": "57db07f736c771b9",
    "dam_e2": "1aee7bb42cd09ac4",
    "dam_e1_mass": "55b670d43a16727f",
    "dam_e1_smart": "ece388dd1d325cb2",
    "chute_e1": "76e9a66344ed0f35",
    "chute_e2": "28f495bdc76b02fa",
    "island_e1": "b8f6ac0b2b254ca2",
    "island_e2": "68e7c9291ec07089",
    "rain_e1": "a94d4a450643bcd6",
    "tsunami_split": "f2376523a29e63c1",
    "chute_e1_split": "4f6a5c7b5f19ad6d",
    "chute_e2_split": "69a7c53aa0291e2d",
    "island_e1_split": "68af487876c244fd",
    "rain_e1_split": "69fecb6642e23d1c",
    "amr_dam_e1_l3": "eb4b83c392ab80fd",
    "amr_dam_e1_l2_rain": "75c26a14ed11b5ac",
    "amr_dam_e2_l2_smart": "f7295b3cf42f5a0c",
    "amr_hump_e2_l2": "d4d35620842fa2a9",
}


@pytest.mark.parametrize("name", list(RUNS))
def test_fast_bits(name):
    assert digest(name) == DIGESTS[name]


def _moved(engine, dx, dy, **kw):
    """Moving water, a shore and a bump in the middle of a basin at rest, moved by (dx, dy)
    cells against the blocks."""
    n = 96
    rng = np.random.default_rng(11)
    c = cases.hump_walls(n, engine)
    bump = np.zeros((n, n))
    bump[24:72, 24:72] = rng.uniform(0.0, 0.3, (48, 48))
    y, x = np.mgrid[0:n, 0:n]
    bump += 1.4 * np.exp(-((x - 54) ** 2 + (y - 44) ** 2) / 40.0)  # (an island)
    bump[np.hypot(x - 48, y - 48) > 26] = 0.0
    zb = (-1.0 + bump).astype(np.float32)
    eta = 0.4 * np.exp(-((x - 40) ** 2 + (y - 50) ** 2) / 30.0)
    eta[np.hypot(x - 48, y - 48) > 26] = 0.0
    c.zb, c.h = zb, np.maximum(eta - zb, 0.0).astype(np.float32)
    c.u, c.v = (np.where((np.hypot(x - 48, y - 48) < 20) & (c.h > 0), rng.uniform(-1, 1, (n, n)), 0).astype(np.float32)
                for _ in range(2))
    for k in ("zb", "h", "u", "v"):
        setattr(c, k, np.roll(getattr(c, k), (dy, dx), (0, 1)))
    return _set(c, cf=0.01, frictionmodel=-1, **kw)


@pytest.mark.parametrize("engine,kw", [(1, {}), (2, {}), (2, {"doubleprecision": 1})], ids=["e1", "e2", "e2_double"])
def test_fast_results_do_not_depend_on_the_blocks(engine, kw):
    """The same water at other places of the blocks gives the same bits: what is formed as
    half of a pair, on the edge of a block or in its ring has the same roundings."""
    def run(dx, dy):
        f, mesh, loop = make_gpu(_moved(engine, dx, dy, **kw))
        dts = []
        for _ in range(12):
            dts.append(f.flow_step(loop))
            loop.totaltime += dts[-1]
        from bg_flood_b200.mesh import buq_to_grid
        return dts, [np.roll(buq_to_grid(a, mesh), (-dy, -dx), (0, 1)) for a in f.get_state()[1:]]

    ref = run(0, 0)
    for dx, dy in ((5, 3), (8, 1), (1, 8)):
        got = run(dx, dy)
        assert got[0] == ref[0]
        for k, a, b in zip("huv", ref[1], got[1]):
            assert np.array_equal(a, b), (dx, dy, k, int((a != b).sum()))
