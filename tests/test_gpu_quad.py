"""The pair kernels where their split of the work changes: the exact build takes one cell
per thread below 700 blocks and pairs from there on (676 and 729 blocks here), both
bit-identical to the separate one-cell kernels of layout 1; and a device-side run, whose
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
