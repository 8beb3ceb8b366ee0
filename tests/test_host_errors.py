"""The library's host code when a call of the CUDA runtime fails, on the CPU: its own objects
are linked with a stand-in for the runtime (fake_cudart.cpp), whose calls a test lets fail."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import bg_flood_b200._native as native
import bg_flood_b200.build as build
import cases
from bg_flood_b200.flow import BGFError, Loop
from runners import make_gpu, make_gpu_amr

HERE = os.path.dirname(os.path.abspath(__file__))
EINVAL, ECUDA = 1, 2


@pytest.fixture(scope="module")
def fake_lib(tmp_path_factory):
    objs = [os.path.join(build.LIBDIR, o) for _, o, _ in build.SOURCES]
    if not all(os.path.exists(o) for o in objs):
        build.build(force=True)
    out = str(tmp_path_factory.mktemp("fake") / "libfake.so")
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-I", cuda, os.path.join(HERE, "fake_cudart.cpp"), *objs,
                    "-Wl,-Bsymbolic", "-lpthread", "-o", out], check=True)
    l = ctypes.CDLL(out)
    for name, (res, args) in native.SIGNATURES.items():
        getattr(l, name).restype, getattr(l, name).argtypes = res, args
    l.fake_fail.argtypes = [ctypes.c_char_p, ctypes.c_int]
    l.fake_calls.argtypes = [ctypes.c_char_p]
    return l


@pytest.fixture
def fake(fake_lib, monkeypatch):
    monkeypatch.setattr(native, "_lib", fake_lib)
    failing = set()

    def fail(name, nth=1):
        failing.add(name)
        fake_lib.fake_fail(name.encode(), nth)

    fail.calls = lambda name: fake_lib.fake_calls(name.encode())
    fail.graphs = fake_lib.fake_live_graphs
    yield fail
    for name in failing:
        fake_lib.fake_fail(name.encode(), 0)


def _single():
    f, _, loop = make_gpu(cases.hump_walls(64, 1))
    loop.nextoutputtime = 1e30
    loop.dtmax = 1.0
    return f, loop


def _amr(name="amrdam64_e1_l2"):
    g = np.load(os.path.join(HERE, "golden", f"{name}.npz"))
    return make_gpu_amr(cases.amr_dambreak(64, 1, 2), (g["level"], g["nbr"], g["xo"], g["yo"]))


def _raises(status, call):
    with pytest.raises(BGFError) as e:
        call()
    assert e.value.status == status


@pytest.mark.parametrize("call", ["step", "run"])
@pytest.mark.parametrize("mk,name", [(_single, "cudaLaunchKernelExC"), (_amr, "cudaLaunchKernelExC"),
                                     (_amr, "cudaEventRecord"), (_amr, "cudaStreamWaitEvent")],
                         ids=["launch", "amr_launch", "fork_record", "fork_wait"])
def test_a_graph_without_one_of_its_launches_is_not_kept(fake, mk, name, call):
    """A launch, or the fork of the multi-level branches, that fails while a graph is captured:
    the call reports it and the next one builds the graph anew."""
    f, loop = mk()
    go = (lambda: f.flow_step(loop)) if call == "step" else (lambda: f.run(loop, 1e30, maxsteps=2))
    fake("cudaGraphLaunch", 0)
    fake(name)
    _raises(ECUDA, go)
    assert fake.calls("cudaGraphLaunch") == 0 and fake.graphs() == 0
    fake(name, 0)
    fake("cudaStreamBeginCapture", 0)
    go()
    assert fake.calls("cudaStreamBeginCapture") == 1 and fake.calls("cudaGraphLaunch") == 1
    f.close()


def test_a_failed_pool_graph_is_not_kept(fake):
    from bg_flood_b200.pool import ScenarioPool
    f, loop = _single()
    pool = ScenarioPool(cases.hump_walls(64, 1).param, 64, 2)
    pool.admit(f, loop, 1e30, maxsteps=4)
    fake("cudaLaunchKernelExC")
    _raises(ECUDA, lambda: pool.run(4))
    fake("cudaLaunchKernelExC", 0)
    pool.run(4)
    assert fake.graphs() == 0
    pool.close()


@pytest.mark.parametrize("name,nth", [("cudaStreamCreateWithPriority", 1), ("cudaEventCreateWithFlags", 1),
                                      ("cudaEventCreateWithFlags", 2)])
def test_the_second_branch_is_complete_or_absent(fake, name, nth):
    """The stream and the two events of the multi-level fork: after one could not be made, the
    next attempt makes what is missing."""
    f, loop = _amr()  # (its tables once more, on a new handle whose first attempt fails)
    blocks = f.get_blocks()
    f.close()
    from bg_flood_b200.flow import FlowB200
    case = cases.amr_dambreak(64, 1, 2)
    g = np.load(os.path.join(HERE, "golden", "amrdam64_e1_l2.npz"))
    n = len(g["level"])
    f = FlowB200(case.param, n)
    set_blocks = lambda: f.set_blocks(np.arange(n, dtype=np.int32), g["level"], g["nbr"], g["xo"], g["yo"])
    fake(name, nth)
    _raises(ECUDA, set_blocks)
    fake(name, 0)
    set_blocks()
    zero = np.zeros((n, 18, 18))
    f.set_bed(zero)
    f.set_state(zero + 1, zero, zero)
    f.flow_step(loop)
    f.close()


@pytest.mark.parametrize("name,nth", [("cudaGraphInstantiate", 2), ("cudaStreamBeginCapture", 2), ("cudaGraphLaunch", 66)])
def test_a_run_that_fails_in_a_later_batch_keeps_its_progress(fake, name, nth):
    """1024 steps in graphs of 16, then 4 more in graphs of two, whose graph cannot be built or
    launched: the loop is where the device is, and another run goes on from there."""
    f, loop = _single()
    fake(name, nth)
    _raises(ECUDA, lambda: f.run(loop, 1e30, maxsteps=1028))
    done = loop.totaltime
    assert done == (1026.0 if name == "cudaGraphLaunch" else 1024.0)  # (a step is a second here)
    fake(name, 0)
    n = f.run(loop, 1e30, maxsteps=1028 - int(done))
    assert n == 1028 - int(done) and loop.totaltime == 1028.0
    f.close()


def test_graphs_a_run_builds(fake):
    """The graph of 16 steps is built once the runs of a handle would replay it often enough,
    not for a short first run; setting something that drops the graphs starts anew."""
    f, loop = _single()

    def built(steps):
        fake("cudaGraphInstantiate", 0)
        fake("cudaGraphLaunch", 0)
        assert f.run(loop, 1e30, maxsteps=steps) == steps
        return fake.calls("cudaGraphInstantiate"), fake.calls("cudaGraphLaunch")

    assert built(20) == (1, 10)
    assert built(20) == (0, 10)
    assert built(20) == (0, 10)
    assert built(20) == (1, 3)      # (80 steps in all: from here on one of 16 and two of two)
    assert built(33) == (0, 3)
    f.set_rain([0.0, 1e9], [1.0, 1.0])
    assert built(20) == (1, 10)
    f.close()
    f, loop = _single()
    assert built(100) == (2, 8)
    f.close()
