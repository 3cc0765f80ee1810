"""Persistent batches whose models share all physics constants, and batches
where one model differs in a single one of them (step, border width, damping):
every member ends as it does alone, in both roundings."""
import numpy as np
import pytest

from helpers import make_solver
import sgfd
import sgfd.workloads as wl

pytestmark = pytest.mark.gpu

BASE = dict(pml=5, nt=20, quirks=sgfd.QUIRKS_FIXED, damping=sgfd.DAMP_LOGR)
ODD = [dict(), dict(dt=0.0004), dict(pml=7), dict(damping=sgfd.DAMP_REFGPU)]


@pytest.mark.parametrize("arith", [sgfd.ARITH_REF, sgfd.ARITH_FAST], ids=["ref", "fast"])
@pytest.mark.parametrize("odd", ODD, ids=["same", "dt", "pml", "damping"])
def test_members_equal_solo_runs(odd, arith):
    ws = [wl.small_random_case(nx=41, ny=37, nz=35, seed=3, **BASE),
          wl.small_random_case(nx=75, ny=30, nz=44, seed=4, **{**BASE, **odd}),
          wl.small_random_case(nx=33, ny=52, nz=29, seed=5, **BASE)]
    members = []
    try:
        for w in ws:
            w.cfg["arith"] = arith
            members.append(make_solver(w))
        with sgfd.Batch(members) as b:
            b.set_persistent(True)
            b.run(0, 20)
            b.synchronize()
            for w, m in zip(ws, members):
                with make_solver(w) as s:
                    s.run(0, 20)
                    s.synchronize()
                    np.testing.assert_array_equal(m.traces(), s.traces())
                    for k in range(9):
                        np.testing.assert_array_equal(m.field(k), s.field(k), err_msg=sgfd.FIELD_NAMES[k])
    finally:
        for m in members:
            m.close()
