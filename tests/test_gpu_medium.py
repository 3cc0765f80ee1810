"""The per-cell values derived from the medium (shear moduli, damping speeds)
follow a new medium upload: a handle whose medium is replaced runs the new
medium's model, bit for bit the oracle's, for every damping profile and both
upload paths."""
import numpy as np
import pytest

from helpers import make_solver, run_oracle
import sgfd
import sgfd.workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("device_upload", [False, True])
@pytest.mark.parametrize("damping", [sgfd.DAMP_REFGPU, sgfd.DAMP_LOGR, sgfd.DAMP_REFCPU])
def test_second_medium_upload(damping, device_upload):
    import torch
    first = wl.small_random_case(nt=24, damping=damping, seed=7)
    w = wl.small_random_case(nt=24, damping=damping, seed=19)
    o = run_oracle(w)
    with make_solver(first) as s:
        s.run(0, 3)
        s.reset()
        if device_upload:
            dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (w.b, w.lam, w.mu)]
            torch.cuda.synchronize()
            s.set_medium_device(*[a.data_ptr() for a in dev])
        else:
            s.set_medium(w.b, w.lam, w.mu)
        s.set_receivers(w.rec_xyz, w.rec_comp, w.nt)
        s.run(0, w.nt)
        s.synchronize()
        np.testing.assert_array_equal(s.traces(), o.traces().astype(np.float32))
        np.testing.assert_array_equal(s.field(sgfd.VX), o.field(sgfd.VX).astype(np.float32))
