"""Batches of small models, whose z chunks are chosen for the batch and not for
each model: every member ends as it does alone, in graph replays, the
persistent launch and 16-bit storage, with steps left over after the replays."""
import numpy as np
import pytest

from helpers import make_solver
import sgfd
import sgfd.workloads as wl

pytestmark = pytest.mark.gpu

NT = 35                                   # two replays of 16 steps and three steps
EDGES = [(34 + 3 * (i % 5), 30 + 2 * (i % 7), 32 + i % 9) for i in range(20)]


def workload(k):
    nx, ny, nz = EDGES[k]
    return wl.small_random_case(nx=nx, ny=ny, nz=nz, pml=4 + k % 3, nt=NT, seed=k, quirks=sgfd.QUIRKS_FIXED)


@pytest.mark.parametrize("mode", ["graph", "persistent", "f16"])
def test_members_equal_solo_runs(mode):
    storage = sgfd.STORE_F16 if mode == "f16" else sgfd.STORE_F32
    ws = [workload(k) for k in range(len(EDGES))]
    members = [make_solver(w, storage=storage) for w in ws]
    try:
        solo = [m.tile()[2] for m in members]
        with sgfd.Batch(members) as b:
            b.set_persistent(mode == "persistent")
            b.run(0, NT)
            b.synchronize()
        assert [m.tile()[2] for m in members] == solo      # the members keep their own
        for w, m in zip(ws, members):
            with make_solver(w, storage=storage) as s:
                s.run(0, NT)
                s.synchronize()
                np.testing.assert_array_equal(m.traces(), s.traces())
                for f in range(9):
                    np.testing.assert_array_equal(m.field(f), s.field(f), err_msg=sgfd.FIELD_NAMES[f])
    finally:
        for m in members:
            m.close()
