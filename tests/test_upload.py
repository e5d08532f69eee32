"""Uploads and downloads at the sizes where their rows, warps and tile counting
change: any particle order in, the same arrays out, and a consistent sort."""
import numpy as np
import pytest

from helpers import params_16k
from simplefluid_gb300 import SPHSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("where", ["pageable", "pinned", "device"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 257, 2049, 32767, 32768, 32801])
def test_state_comes_back_as_uploaded(n, where):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    arrays = [rng.random((n, 3)).astype(np.float32), rng.normal(size=(n, 3)).astype(np.float32)]  # no order at all
    arrays[1][0] = np.inf, -0.0, np.nan
    if where != "pageable":
        arrays = [torch.from_numpy(a) for a in arrays]
        arrays = [a.pin_memory().numpy() if where == "pinned" else a.cuda() for a in arrays]
    with SPHSolver(params_16k()) as s:
        for _ in range(2):  # the second finds the counters as the first left them
            if where == "device":
                out = [torch.empty_like(a) for a in arrays]
                s.setParticlesDevice(*arrays)
                s.getStateDevice(*out)
                s.synchronize()
            else:
                s.setParticles(*arrays)
                out = s.getState()
            for a, b in zip(arrays, out):
                a, b = (x.cpu().numpy() if where == "device" else x for x in (a, b))
                assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
            report = s.checkState()
            assert not report["unsorted"] and not report["cell_table_mismatch"] and not report["bad_ids"], report
