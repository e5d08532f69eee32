"""Which kernels a sub-step launches: by the size of the scene, unless the caller chose them."""
import pytest

from helpers import params_16k
from simplefluid_gb300 import SPHSolver
from test_contexts import cloud

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
