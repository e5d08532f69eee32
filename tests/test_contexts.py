"""Many contexts with long queues of sub-steps that change their graphs while
they are queued: every context's state is that of a run by itself."""

import threading

import numpy as np
import pytest

from helpers import params_16k
from simplefluid_gb300 import SPHSolver

pytestmark = pytest.mark.gpu


def cloud(n, seed, extent=0.35):
    rng = np.random.default_rng(seed)
    return (0.05 + extent * rng.random((n, 3))).astype(np.float32)


def same_bits(a, b):
    assert all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in zip(a, b))


def test_graphs_given_up_while_they_are_queued():
    """Calls of different lengths, new sizes and new frame times without a wait in between: more graphs than are kept
    until the stream is waited for."""
    prm = params_16k(timeStep=1e-5)
    with SPHSolver(prm) as s, SPHSolver(prm) as one:
        for n in (3000, 2500):
            s.setParticles(cloud(n, n))
            one.setParticles(cloud(n, n))
            steps = 0
            for k in range(6, 18):
                for _ in range(3):  # the third equal call makes a graph of that many
                    s.step(k)
                steps += 3 * k
            for f in (2, 3, 4):
                steps += s.advanceFrames(1, f * 1e-5, 100)[1]
            for _ in range(steps):
                one.advanceFrame()
            same_bits(s.getState(), one.getState())


def test_hundreds_of_contexts_in_bursts_and_in_turn():
    """160 contexts stepped in bursts, in turn and in bursts again, nothing waited for until the end."""
    prm = params_16k(timeStep=1e-5)
    state = [cloud(1500 + 37 * k, k) for k in range(160)]
    ctxs = [SPHSolver(prm) for _ in state]
    try:
        for s, x in zip(ctxs, state):
            s.setParticles(x)
        steps = 0
        for k in (5, 1, 5):
            for s in ctxs:
                for _ in range(5):
                    s.step(k)
            for _ in range(6):
                for s in ctxs:
                    s.step(k)
            steps += 11 * k
        got = [s.getState() for s in ctxs]
    finally:
        for s in ctxs:
            s.close()
    for k in range(0, 160, 20):
        with SPHSolver(prm) as one:
            one.setParticles(state[k])
            for _ in range(steps):
                one.advanceFrame()
            same_bits(got[k], one.getState())


def test_device_frames_on_many_threads():
    """Frames of 12 contexts at once (more than run their sub-steps in runs) equal those of one after the other."""
    prm = params_16k(timeStep=2e-4)
    state = [cloud(900 + 61 * k, k) for k in range(12)]

    def frames(s):
        return [s.advanceFrames(2, f * 2e-4, 1000) for f in (7.5, 21.0, 21.0, 40.0)]

    want = []
    for x in state:
        with SPHSolver(prm) as s:
            s.setParticles(x)
            want.append((frames(s), s.getState()))
    ctxs = [SPHSolver(prm) for _ in state]
    try:
        for s, x in zip(ctxs, state):
            s.setParticles(x)
        times = [None] * 12

        def run(k):
            times[k] = frames(ctxs[k])

        threads = [threading.Thread(target=run, args=(k,)) for k in range(12)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        for s, t, (want_times, want_state) in zip(ctxs, times, want):
            assert t == want_times
            same_bits(s.getState(), want_state)
    finally:
        for s in ctxs:
            s.close()
