"""The pair kernels where their split of the work changes: the exact build takes one cell
per thread below 700 blocks and pairs from there on (676 and 729 blocks here; moving water on
729), both bit-identical to the separate one-cell kernels of layout 1; and a device-side run, whose
graphs hold two steps or (long runs) 16, gives the bits of single steps: for step counts
around that length, from either parity of the time slots, and over several runs."""
import numpy as np
import pytest

import cases
from runners import interior, make_gpu

pytestmark = pytest.mark.gpu


def _steps(case, layout, nsteps, graph=False):
    case.param.fastmath = 0
    f, _, loop = make_gpu(case)
    f.set_kernel_layout(layout)
    if graph:
        loop.nextoutputtime = 1e30
        for n in nsteps:
            if n:
                assert f.run(loop, 1e30, maxsteps=n) == n
            else:  # one single step
                loop.totaltime += f.flow_step(loop)
        return loop.dt, f.get_state()
    loop.nextoutputtime = 1e30
    for _ in range(nsteps):
        dt = f.flow_step(loop)
        loop.totaltime += dt
    return dt, f.get_state()


def _same(a, b):
    assert a[0] == b[0]
    for k, x, y in zip("zs h u v".split(), a[1], b[1]):
        assert np.array_equal(interior(x), interior(y)), k


@pytest.mark.parametrize("n", [416, 432])
@pytest.mark.parametrize("mk", [lambda n: cases.conical_island(n, 1), lambda n: cases.conical_island(n, 2),
                                lambda n: cases.rain_on_terrain(n, 1)], ids=["island_e1", "island_e2", "rain_e1"])
def test_exact_lanes(mk, n):
    _same(_steps(mk(n), 1, 6), _steps(mk(n), 2, 6))


@pytest.mark.parametrize("runs", [[1], [2], [15], [16], [17], [33], [64], [65], [81], [0, 64], [0, 79, 3], [20, 20, 20, 20, 7],
                                  [70, 0, 70, 0, 18]], ids=str)
def test_run_lengths(runs):
    """(0 stands for a single step, which changes the parity)"""
    n = sum(max(k, 1) for k in runs)
    _same(_steps(cases.conical_island(48, 1), 2, n), _steps(cases.conical_island(48, 1), 2, runs, graph=True))


# ---------------------------------------------------------------- exact pairs, moving water
# 27 x 27 blocks (the tsunami 875), so that the exact build's kernels run pairs

def _bumpy(case, seed=4):
    """Random velocities on the wet cells and a rough bed: wetting and drying everywhere."""
    rng = np.random.default_rng(seed)
    ny, nx = case.zb.shape
    case.zb = (case.zb + 0.3 * case.h.max() * rng.uniform(-1, 1, (ny, nx)) ** 3).astype(np.float32)
    wet = case.h > 0
    case.u, case.v = (np.where(wet, 0.3 * rng.standard_normal((ny, nx)), 0.0).astype(np.float32) for _ in range(2))
    return case


def _split(case):
    case.param.splitprecision = 1
    return case


PAIRS = {
    "gauss_e1_absorbing": lambda: cases.gauss(432, 1, 3),
    "gauss_e2_absorbing": lambda: cases.gauss(432, 2, 3),
    "dam_e1": lambda: cases.dam_break(432, 1),
    "dam_e2": lambda: cases.dam_break(432, 2),
    "island_e1": lambda: _bumpy(cases.conical_island(432, 1)),
    "rain_e1": lambda: cases.rain_on_terrain(432, 1),
    "dam_e1_split": lambda: _split(cases.dam_break(432, 1)),
    "dam_e2_split": lambda: _split(cases.dam_break(432, 2)),
    "tsunami_split": lambda: _split(cases.ensemble_member(3, 2024, 740, 900)),
}


def _moving(case, layout, nsteps=30, grid=0, mesh=None):
    from bg_flood_b200.flow import Loop, build_model
    case.param.fastmath = 0
    f, mesh = build_model(case.param, case.zb, case.h, case.u, case.v, rain=case.rain, mesh=mesh)
    assert mesh.nblk >= 700
    f.set_kernel_layout(layout)
    f.set_grid(grid)
    loop = Loop(nextoutputtime=case.nextoutputtime)
    f.init_dt(loop)
    for _ in range(nsteps):
        dt = f.flow_step(loop)
        loop.totaltime += dt
    return dt, f.get_state()


@pytest.mark.parametrize("name", list(PAIRS))
def test_exact_pairs_moving_water(name):
    a, b = (_moving(PAIRS[name](), layout) for layout in (1, 2))
    assert np.abs(interior(a[1][2])).max() > 0 and np.abs(interior(a[1][3])).max() > 0
    _same(a, b)


@pytest.mark.parametrize("engine", [1, 2])
def test_exact_pairs_masked_mesh(engine):
    """A mesh with holes and a ragged edge: the neighbours come from the tables."""
    from bg_flood_b200.mesh import uniform_mesh
    mk = lambda: _bumpy(cases.gauss(480, engine, 3))
    present = np.random.default_rng(2).uniform(size=(30, 30)) > 0.15
    mesh = lambda: uniform_mesh(480, 480, mk().param.dx, present)
    _same(_moving(mk(), 1, mesh=mesh()), _moving(mk(), 2, mesh=mesh()))


@pytest.mark.parametrize("grid", [7, 100])
def test_exact_pairs_persistent_grid(grid):
    _same(_moving(PAIRS["dam_e1"](), 1, 12), _moving(PAIRS["dam_e1"](), 2, 12, grid))


@pytest.mark.parametrize("split", [0, 1])
def test_exact_pairs_in_a_pool(split):
    """Three members of 256 blocks: pairs in the pool of 768, one cell per thread alone."""
    from bg_flood_b200.pool import ScenarioPool

    def mk(k):
        case = [lambda: cases.dam_break(256, 1), lambda: cases.gauss(256, 1, 3), lambda: cases.dam_break(256, 1, seed=8)][k]()
        case.param.fastmath, case.param.splitprecision = 0, split
        return case

    steps = [20, 13, 30]
    alone = []
    for k, n in enumerate(steps):
        f, _, loop = make_gpu(mk(k))
        f.run(loop, 1e30, maxsteps=n)
        alone.append(f.get_state())
        f.close()
    built = [make_gpu(mk(k)) for k in range(3)]
    pool = ScenarioPool(mk(0).param, 768, 3)
    slots = [pool.admit(f, lp, 1e30, maxsteps=n) for (f, _, lp), n in zip(built, steps)]
    assert pool.run(64) == 0
    for slot, st in zip(slots, alone):
        assert np.array_equal(np.asarray(pool.depth(slot, 256), np.float64).astype(np.float32),
                              interior(st[1]).astype(np.float32))
    pool.close()
