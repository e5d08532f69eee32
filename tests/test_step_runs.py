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
