"""More receivers on one plane of a tile than its CTA has threads, for every
tile shape and in the persistent batch, in the interior, in the border and on
both sides of a z-chunk line: traces equal the oracle's bit for bit."""
import numpy as np
import pytest

from helpers import make_solver, run_oracle
import sgfd
import sgfd.workloads as wl

pytestmark = pytest.mark.gpu

TILES = [(32, 8, 0), (32, 8, 4), (32, 16, 4), (64, 8, 4)]
THREADS = 256
PLANES = (5, 12, 13, 24)


def workload(per_plane):
    """per_plane receivers on each plane, all in the first 32 x 8 computed cells (the first tile of every shape)."""
    w = wl.small_random_case(nx=71, ny=33, nz=30, pml=4, nt=12, quirks=sgfd.QUIRKS_FIXED, damping=sgfd.DAMP_LOGR)
    rng = np.random.Generator(np.random.PCG64(5))
    n = per_plane * len(PLANES)
    xyz = np.stack([rng.integers(5, 37, n), rng.integers(5, 13, n), np.repeat(PLANES, per_plane)], 1)
    order = rng.permutation(n)
    w.rec_xyz = xyz[order].astype(np.int32)
    w.rec_comp = rng.integers(0, 9, n).astype(np.int32)
    return w


@pytest.fixture(scope="module", params=[THREADS, THREADS + 1, 3 * THREADS - 1])
def case(request):
    w = workload(request.param)
    return w, run_oracle(w).traces().astype(np.float32)


@pytest.mark.parametrize("tile", TILES, ids=lambda t: "%dx%d_chunk%d" % t)
def test_traces_equal_the_oracle(case, tile):
    w, want = case
    with make_solver(w) as s:
        s.set_tile(*tile)
        s.run(0, w.nt)
        s.synchronize()
        np.testing.assert_array_equal(s.traces(), want)


def test_traces_in_a_persistent_batch(case):
    w, want = case
    with make_solver(w) as a, make_solver(w) as b, sgfd.Batch([a, b]) as batch:
        batch.set_persistent(True)
        batch.run(0, w.nt)
        batch.synchronize()
        for s in (a, b):
            np.testing.assert_array_equal(s.traces(), want)
