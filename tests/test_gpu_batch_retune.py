"""A member's launch shape set between two runs of a batch, without waiting for
the first: the first run's steps are not disturbed, the second takes the new
shape, and every member ends as it does alone."""
import numpy as np
import pytest

from helpers import make_solver
import sgfd
import sgfd.workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["graph", "persistent"])
def test_chunk_set_between_runs(mode):
    nt = 120
    ws = [wl.small_random_case(nx=50 + 3 * k, ny=44, nz=60 - k, pml=5, nt=nt, seed=k) for k in range(4)]
    members = [make_solver(w) for w in ws]
    try:
        with sgfd.Batch(members) as b:
            b.set_persistent(mode == "persistent")
            for it, n, zc in ((0, 64, 9), (64, 32, 3), (96, 24, 0)):
                b.run(it, n)
                for m in members:
                    m.set_zchunk(zc)
            b.synchronize()
        for w, m in zip(ws, members):
            with make_solver(w) as s:
                s.run(0, nt)
                s.synchronize()
                np.testing.assert_array_equal(m.traces(), s.traces())
                for f in range(9):
                    np.testing.assert_array_equal(m.field(f), s.field(f), err_msg=sgfd.FIELD_NAMES[f])
    finally:
        for m in members:
            m.close()
