"""The automatic z chunk on both sides of each line of its rule (one wave,
about four waves, many waves): traces and fields equal those of a fixed
16-plane chunk bit for bit, for FP32 and 16-bit storage."""
import numpy as np
import pytest

from helpers import make_solver
import sgfd
import sgfd.workloads as wl

pytestmark = pytest.mark.gpu

# extents whose automatic chunk is one plane, a few planes, one wave of the
# longest such chunk, several waves of short chunks, and the 16-plane floor
GRIDS = [(30, 24, 22), (64, 60, 66), (100, 100, 99), (122, 118, 121), (230, 210, 130)]


@pytest.mark.parametrize("storage", [sgfd.STORE_F32, sgfd.STORE_F16])
@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "%dx%dx%d" % g)
def test_automatic_chunk(grid, storage):
    nx, ny, nz = grid
    w = wl.small_random_case(nx=nx, ny=ny, nz=nz, pml=5, nt=8, nrec=40, quirks=sgfd.QUIRKS_FIXED)
    got = []
    for zc in (0, 16):
        with make_solver(w, storage=storage) as s:
            s.set_zchunk(zc)
            assert 1 <= s.tile()[2] <= nz - 10
            s.run(0, w.nt)
            s.synchronize()
            got.append([s.traces(), s.field(sgfd.VZ), s.field(sgfd.TXY)])
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
