"""The small-scene (team) passes and the paired force gather against the
one-thread passes and the oracle: the same bits at every size and state where
their tiles, lists or number ranges could go wrong."""
import numpy as np
import pytest

from helpers import params_16k
from simplefluid_gb300 import SPHSolver
from simplefluid_gb300 import _capi as C

pytestmark = pytest.mark.gpu


def block(n, seed, spacing=0.02, jitter=0.3):
    """n particles of a jittered lattice (y slowest) in a corner of the unit box."""
    a = 1
    while a * a * 2 * a < n:
        a += 1
    t = np.arange(n)
    x = np.stack([t % a, t // (a * a), (t // a) % a], 1) * spacing + spacing / 2
    rng = np.random.default_rng(seed)
    x = x + jitter * spacing * (2.0 * rng.random((n, 3)) - 1.0)
    return x.astype(np.float32), rng.normal(scale=0.3, size=(n, 3)).astype(np.float32)


def one_thread(s, prefetch=4, list_mode=C.SF_LIST_TILE):
    """128-thread density blocks select the one-thread passes."""
    t = s.getTuning()
    t.density_block, t.force_block, t.prefetch, t.list_mode = 128, 128, prefetch, list_mode
    s.setTuning(t)


def run(prm, pos, vel, tune=None, steps=2):
    with SPHSolver(prm) as s:
        s.setParticles(pos, vel)
        if tune:
            tune(s)
        rho, prs = s.computeDensity()
        acc = s.computeAccel()
        overflows = s.checkState()["list_overflow"]
        s.step(steps)
        return rho, prs, acc, overflows, *s.getState()


def same(a, b):
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)  # NaN equals NaN


@pytest.mark.parametrize("cells", [1, 2, 3])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 2049])
def test_small_sizes_equal_one_thread_passes_and_oracle(oracle, n, cells):
    prm = params_16k(cellsPerH=cells)
    pos, vel = block(n, n)
    got = run(prm, pos, vel)
    same(got, run(prm, pos, vel, one_thread))
    st = oracle.State(pos, vel)
    st.step(prm.to_c(), 2)
    opos, ovel = st.original_order()
    assert np.array_equal(got[-2].view(np.uint32), opos.view(np.uint32))
    assert np.array_equal(got[-1].view(np.uint32), ovel.view(np.uint32))


@pytest.mark.parametrize("n", [32767, 32768, 57343, 57344])
def test_sizes_where_the_passes_change(n):
    r = 0.005
    prm = params_16k(particleRadius=r, kernelRadius=4 * r)
    pos, vel = block(n, n, spacing=2 * r)
    same(run(prm, pos, vel), run(prm, pos, vel, one_thread))


@pytest.mark.parametrize("cells", [1, 2, 3])
def test_dense_places(cells):
    """Lists over 64 neighbours, rows over 32 candidates, coincident particles and one that is not a number."""
    rng = np.random.default_rng(7)
    pos, vel = block(3000, 3)
    pos[100:140] = pos[50]  # coincident
    pos[200:420] = pos[60] + 1e-3 * rng.random((220, 3))  # one crowded cell
    pos[500:560] = pos[70] + 0.004 * rng.random((60, 3))  # about one full list
    pos = pos.astype(np.float32)
    prm = params_16k(cellsPerH=cells, timeStep=1e-6)
    got = run(prm, pos, vel)
    assert got[3] > 0
    same(got, run(prm, pos, vel, one_thread))
    pos[700] = np.nan
    same(run(prm, pos, vel), run(prm, pos, vel, one_thread))


@pytest.mark.parametrize("h", [1e-6, 3.0e-6, 2.0 ** -17, 2.0 ** -5, 0.04, 0.0371, 1e6])
def test_root_and_quotient_at_every_scale(h):
    """The paired gather's root and quotient against the compiler's (rescans of the candidate cells): kernel radii in
    and out of its range, among them powers of two, with coincident and nearly coincident particles."""
    pos, vel = block(1500, 11)
    prm = params_16k(kernelRadius=h, particleRadius=h / 4, boxMax=(25 * h,) * 3, timeStep=1e-9 * h)
    pos = (pos * (h / 0.04)).astype(np.float32)
    pos[10:14] = pos[9]
    pos[20:24] = [[0, 0, 0], [1e-15 * h, 0, 0], [0, 2e-20, 1e-21], [0, 1e-9 * h, 0]]
    vel = (vel * h).astype(np.float32)
    want = run(prm, pos, vel, lambda s: one_thread(s, list_mode=C.SF_LIST_NONE))
    for tune in (None, lambda s: one_thread(s, 2), lambda s: one_thread(s, 2, C.SF_LIST_TILE16)):
        got = run(prm, pos, vel, tune)
        for k in (0, 1, 2, 4, 5):
            np.testing.assert_array_equal(got[k], want[k])


@pytest.mark.parametrize("seed_scale", [1.0, 1e-20, 1e-33, 1e-38])
@pytest.mark.parametrize("h", [0.04, 2.0 ** -5, 2048.0])
def test_adjoint_pairs_equal_oracle(oracle, h, seed_scale):
    """The adjoint's paired force terms: kernel radii in and out of their range, adjoints down to numbers whose
    quotients underflow (most particles have none), coincident and nearly coincident particles."""
    n = 700
    pos, vel = block(n, 5)
    pos = (pos * (h / 0.04)).astype(np.float32)
    pos[10:12] = pos[9]
    pos[20] = pos[21] + np.float32(1e-6 * h)
    vel = (vel * h).astype(np.float32)
    prm = params_16k(kernelRadius=h, particleRadius=h / 4, boxMax=(25 * h,) * 3, timeStep=1e-6)
    rng = np.random.default_rng(3)
    gx = np.zeros((n, 3), np.float32)
    gx[::50] = (seed_scale * rng.normal(size=gx[::50].shape)).astype(np.float32)
    with SPHSolver(prm) as s:
        s.setParticles(pos, vel)
        s.forward(3, 2)
        dx0, dv0, _, _ = s.adjoint(gx)
    want = oracle.adjoint(prm.to_c(), pos, vel, 3, gx, ckpt=2, dtype=np.float32)
    np.testing.assert_array_equal(dx0, want[0])
    np.testing.assert_array_equal(dv0, want[1])


@pytest.mark.parametrize("n", [81919, 81920, 196607, 196608, 262143, 262144])
def test_sizes_where_the_blocks_and_launches_change(n):
    r = 0.0025
    prm = params_16k(particleRadius=r, kernelRadius=4 * r)
    pos, vel = block(n, n, spacing=2 * r)

    def blocks_256(s):
        t = s.getTuning()
        t.density_block = t.force_block = 256
        s.setTuning(t)

    same(run(prm, pos, vel), run(prm, pos, vel, blocks_256))


@pytest.mark.parametrize("cells", [1, 2, 3])
@pytest.mark.parametrize("spacing", [0.0165, 0.0145, 0.0125, 0.0105])
def test_more_neighbours_than_a_list_holds(spacing, cells):
    """Lattices of about 60, 88, 137 and 232 neighbours: lists that just overflow, sums in up to four rounds, rows of
    more than 32, 64 and 96 candidates."""
    pos, vel = block(3001, 9, spacing=spacing, jitter=0.2)
    got = run(params_16k(cellsPerH=cells, timeStep=1e-6), pos, vel)
    assert got[3] > 0
    same(got, run(params_16k(cellsPerH=cells, timeStep=1e-6), pos, vel, one_thread))
