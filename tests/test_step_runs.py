"""Sub-steps are queued one by one, as single graphs or in runs: the same state whatever the calls."""
import numpy as np
import pytest

from helpers import params_16k
from simplefluid_gb300 import SPHSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("adaptive", [False, True])
@pytest.mark.parametrize("calls", [[13], [5, 5, 3], [1, 12], [4, 9], [2, 2, 9], [33, 13, 1]])
def test_any_split_of_the_steps_gives_the_same_state(calls, adaptive):
    rng = np.random.default_rng(1)
    g = np.stack(np.meshgrid(*[np.arange(k) for k in (9, 12, 11)], indexing="ij"), -1).reshape(-1, 3)
    pos = ((g + 0.5) * 0.02 + 0.002 * rng.random(g.shape)).astype(np.float32)
    vel = rng.normal(scale=0.5, size=pos.shape).astype(np.float32)
    prm = params_16k(adaptiveTimeStep=adaptive, timeStep=5e-4)
    with SPHSolver(prm) as s, SPHSolver(prm) as one:
        for upload in (pos, pos[:900]):  # a new size drops the graphs
            s.setParticles(upload, vel[:len(upload)])
            one.setParticles(upload, vel[:len(upload)])
            for k in calls:
                s.step(k)
                for _ in range(k):
                    one.advanceFrame()
                for a, b in zip(s.getState(), one.getState()):
                    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("adaptive", [False, True])
@pytest.mark.parametrize("max_substeps", [1, 4, 5, 16, 17, 21, 10000])
@pytest.mark.parametrize("steps", [0.5, 3.5, 4.0, 5.0, 16.0, 17.5, 37.0])
def test_a_frame_ends_where_its_sub_steps_do(steps, max_substeps, adaptive):
    rng = np.random.default_rng(2)
    pos = (0.1 + 0.2 * rng.random((700, 3))).astype(np.float32)
    vel = rng.normal(scale=4.0 if adaptive else 0.5, size=pos.shape).astype(np.float32)  # CFL-limited: dt below the step
    prm = params_16k(adaptiveTimeStep=adaptive, timeStep=2e-3)
    frame = steps * 2e-3
    with SPHSolver(prm) as s, SPHSolver(prm) as one:
        s.setParticles(pos, vel)
        one.setParticles(pos, vel)
        for _ in range(2):
            t, k = s.advanceFrames(1, frame, max_substeps)
            acc, n = np.float32(0.0), 0
            while float(acc) < frame and n < max_substeps:
                acc = np.float32(acc + np.float32(one.advanceFrame()))
                n += 1
            assert k == n and np.float32(t) == acc
            for a, b in zip(s.getState(), one.getState()):
                assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


@pytest.mark.parametrize("calls", [[7] * 5 + [3, 7, 9, 9, 9, 9, 7], [40] * 4 + [6], [300]])
def test_repeated_and_long_calls_give_the_same_state(calls):
    rng = np.random.default_rng(3)
    pos = (0.1 + 0.3 * rng.random((900, 3))).astype(np.float32)
    prm = params_16k(timeStep=5e-4)
    with SPHSolver(prm) as s, SPHSolver(prm) as one:
        for upload in (pos, pos[:800]):
            s.setParticles(upload)
            one.setParticles(upload)
            for k in calls:
                s.step(k)
            for _ in range(sum(calls)):
                one.advanceFrame()
            for a, b in zip(s.getState(), one.getState()):
                assert np.array_equal(a.view(np.uint32), b.view(np.uint32))


def test_contexts_stepped_in_turn_give_the_state_of_one_alone():
    """Four small scenes and the calls that decide whether they share the GPU."""
    rng = np.random.default_rng(4)
    prm = params_16k(particleRadius=0.005, kernelRadius=0.02)
    pos = [(0.05 + 0.35 * rng.random((25000, 3))).astype(np.float32) for _ in range(4)]
    alone = []
    for p in pos:
        with SPHSolver(prm) as s:
            s.setParticles(p)
            s.step(14)
            alone.append(s.getState())
    solvers = [SPHSolver(prm) for _ in pos]
    try:
        for s, p in zip(solvers, pos):
            s.setParticles(p)
        for _ in range(9):  # in turn: from the fifth round on as sharing
            for s in solvers:
                s.step(1)
        for s in solvers:  # each by itself again
            for _ in range(5):
                s.step(1)
        for s, want in zip(solvers, alone):
            for a, b in zip(s.getState(), want):
                assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    finally:
        for s in solvers:
            s.close()
