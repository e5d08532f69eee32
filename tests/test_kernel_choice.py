"""Which kernels a sub-step launches: by the size of the scene, unless the caller chose them."""
import os
import subprocess
import sys
import threading

import pytest

from helpers import params_16k
from simplefluid_gb300 import SPHSolver
from simplefluid_gb300 import _capi as C
from test_contexts import cloud, same_bits

pytestmark = pytest.mark.gpu

STAGES = ["density", "force_integrate", "scan", "scatter", "rank_gather"]


def kernels(s):
    k = s.stageKernels()
    assert list(k) == STAGES
    return tuple(k.values())


def test_stages_report_their_kernels():
    with SPHSolver(params_16k()) as s:
        assert kernels(s) == ("",) * 5
        s.setParticles(cloud(2000, 1))
        assert kernels(s) == ("density_team", "force_team", "scan", "", "list_gather")
    with SPHSolver(params_16k(cellsPerH=1)) as s:
        s.setParticles(cloud(2000, 1))
        assert kernels(s)[2:] == ("scan", "scatter", "rank_gather")


@pytest.mark.parametrize("n", [2000, 40000, 100000, 300000])
def test_an_explicit_choice_is_taken_at_every_size(n):
    """Also the blocks that sf_get_tuning reports before any choice; the state is the same."""
    prm = params_16k(particleRadius=0.0025, kernelRadius=0.01)
    pos = cloud(n, n, 0.3)
    with SPHSolver(prm) as s:
        s.setParticles(pos)
        s.step(2)
        want = s.getState()
        for density, force, gather in ((256, 128, 2), (256, 128, 4), (128, 256, 4), (256, 256, 2)):
            s.setTuning(C.sf_tuning(C.SF_LIST_TILE, density, force, gather))
            s.setParticles(pos)
            assert kernels(s)[:2] == (f"density_{density}", f"force_{force}" + ("_gather4" if gather == 4 else ""))
            s.step(2)
            same_bits(s.getState(), want)


def test_frames_reserve_the_l2_window():
    """A program that only runs frames gets the window it asked for (in a process of its own: the reservation is the
    process's)."""
    code = """
import ctypes
import numpy as np
from simplefluid_gb300 import SPHParameters, SPHSolver
from simplefluid_gb300 import _capi as C

def reserved():
    size = ctypes.c_size_t()
    assert ctypes.CDLL("libcuda.so.1").cuCtxGetLimit(ctypes.byref(size), 6) == 0  # persisting L2
    return size.value

s = SPHSolver(SPHParameters(particleRadius=0.0025, kernelRadius=0.01))
s.setTuning(C.sf_tuning(C.SF_LIST_TILE, 256, 128, 2, 1))
s.setParticles(np.random.default_rng(1).random((1500000, 3)).astype(np.float32))
assert reserved() < 1500000 * 32  # the device's default
s.advanceFrames(1, 2e-4, 10)
assert reserved() >= 1500000 * 32, reserved()
s.close()
"""
    out = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120,
                         cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert out.returncode == 0, out.stderr[-2000:]


def test_the_sort_follows_the_grid_not_its_history():
    """The same cells as one per h and as two per 2h: the kernels and the state of a context that switches, with and
    without particles, are those of a new one."""
    both = [params_16k(kernelRadius=h, cellsPerH=k) for h, k in ((0.04, 1), (0.08, 2))]
    pos = cloud(3000, 3)
    with SPHSolver(both[1]) as s:
        for prm, other in (both, both[::-1], both):
            s.setParams(prm)
            s.setParticles(pos)
            s.setParams(other)
            s.setParams(prm)
            with SPHSolver(prm) as new:
                new.setParticles(pos)
                assert s.gridDims() == new.gridDims()
                assert kernels(s) == kernels(new)
                s.step(3)
                new.step(3)
                same_bits(s.getState(), new.getState())


@pytest.mark.parametrize("cells", [1, 2, 3])
@pytest.mark.parametrize("ratio,team", [(4.0, True), (4.9, True), (5.0, False), (8.0, False)])
def test_no_teams_where_the_lists_overflow_at_rest(ratio, team, cells):
    with SPHSolver(params_16k(kernelRadius=0.01 * ratio, cellsPerH=cells)) as s:
        s.setParticles(cloud(2000, 1))
        assert kernels(s)[:2] == (("density_team", "force_team") if team else ("density_256", "force_128_gather4"))


@pytest.fixture
def four():
    """Four scenes of 30,000 particles: any two of them fill the GPU."""
    prm = params_16k(particleRadius=0.005, kernelRadius=0.02)
    solvers = [SPHSolver(prm) for _ in range(4)]
    for k, s in enumerate(solvers):
        s.setParticles(cloud(30000, k))
        s.step(1)
        s.synchronize()
    yield solvers
    for s in solvers:
        s.close()


def teams(s):
    return kernels(s)[0] == "density_team"


def test_contexts_that_keep_the_gpu_busy_take_one_thread_per_particle(four):
    for _ in range(20):
        for s in four:
            s.step(20)
    assert not any(teams(s) for s in four)
    for s in four:
        s.synchronize()
    four[0].step(1)
    assert teams(four[0])


@pytest.mark.parametrize("wait", ["synchronize", "device"])
def test_contexts_waited_for_in_turn_keep_their_teams(four, wait):
    torch = pytest.importorskip("torch")
    big = SPHSolver(params_16k(particleRadius=0.0025, kernelRadius=0.01))
    big.setParticles(cloud(300000, 9, 0.4))
    try:
        for _ in range(8):
            for s in (big, *four):
                s.step(2)
                s.synchronize() if wait == "synchronize" else torch.cuda.synchronize()
                assert s is big or teams(s)
    finally:
        big.close()


def test_frames_of_several_threads_take_one_thread_per_particle(four):
    for _ in range(2):  # one after the other on this thread
        for s in four:
            s.advanceFrames(1, 3e-4, 100)
            assert teams(s)
    for _ in range(2):
        threads = [threading.Thread(target=s.advanceFrames, args=(1, 3e-4, 100)) for s in four]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not any(teams(s) for s in four)
    for s in four:  # this thread's again
        s.advanceFrames(1, 3e-4, 100)
    assert teams(four[3])
