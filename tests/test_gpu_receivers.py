"""Receiver recording of the z-marching kernels where a tile's plane holds more
receivers than the CTA has threads, several receivers per cell, every plane of
a column, and planes on both sides of a z-chunk border: traces equal the
oracle's bit for bit."""
import numpy as np
import pytest

from helpers import make_solver, run_oracle
import sgfd
import sgfd.workloads as wl

pytestmark = pytest.mark.gpu

TILES = [(32, 8, 0), (32, 8, 3), (32, 16, 5), (64, 8, 4)]


def workload(nrec_plane):
    w = wl.small_random_case(nx=71, ny=33, nz=30, pml=4, nt=12, quirks=sgfd.QUIRKS_FIXED, damping=sgfd.DAMP_LOGR)
    rng = np.random.Generator(np.random.PCG64(11))
    pts = []
    for z in (5, 11, 12, 24):      # whole planes, cells repeated
        x, y = rng.integers(5, 66, nrec_plane), rng.integers(5, 28, nrec_plane)
        pts.append(np.stack([x, y, np.full(nrec_plane, z)], 1))
    col = np.array([[37, 14, z] for z in range(30)])          # a column through the whole GRID, frame included
    one = np.array([[20, 9, 15]] * 9)                         # nine components of one cell
    xyz = np.concatenate(pts + [col, one]).astype(np.int32)
    comp = np.concatenate([rng.integers(0, 9, 4 * nrec_plane), np.arange(30) % 9, np.arange(9)]).astype(np.int32)
    order = rng.permutation(len(xyz))
    w.rec_xyz, w.rec_comp = xyz[order], comp[order]
    return w


@pytest.mark.parametrize("tile", TILES, ids=lambda t: "%dx%d_chunk%d" % t)
@pytest.mark.parametrize("nrec_plane", [1, 700])
def test_dense_receivers_equal_the_oracle(nrec_plane, tile):
    w = workload(nrec_plane)
    o = run_oracle(w)
    with make_solver(w) as s:
        s.set_tile(*tile)
        s.run(0, w.nt)
        s.synchronize()
        np.testing.assert_array_equal(s.traces(), o.traces().astype(np.float32))


def test_dense_receivers_in_a_persistent_batch():
    w = workload(700)
    o = run_oracle(w)
    with make_solver(w) as a, make_solver(w) as b:
        with sgfd.Batch([a, b]) as batch:
            batch.set_persistent(True)
            batch.run(0, w.nt)
            batch.synchronize()
            for s in (a, b):
                np.testing.assert_array_equal(s.traces(), o.traces().astype(np.float32))
