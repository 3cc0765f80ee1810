"""Half steps in parts on both sides of the line below which the inner part runs
with the outer one (less than one wave of CTAs), and a model in more slabs than
three: the same bits as whole steps."""
import numpy as np
import pytest

from helpers import make_solver
import sgfd
import sgfd.slabs as sl
import sgfd.workloads as wl

pytestmark = pytest.mark.gpu


def inner_launch(nx, ny, nz, chunk):
    """Whether the inner chunks (5 or more planes from both ends) make one wave of three CTAs per SM."""
    import torch
    tiles = -(-(nx - 10) // 32) * -(-(ny - 10) // 8)
    inner = sum(1 for z in range(0, nz - 10, chunk) if z >= 5 and min(z + chunk, nz - 10) <= nz - 15)
    return tiles * inner >= 3 * torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("nx,ny,nz,chunk", [(75, 60, 44, 1), (75, 60, 44, 4), (234, 170, 40, 3), (39, 35, 24, 2)])
def test_parts_equal_steps(nx, ny, nz, chunk):
    own = inner_launch(nx, ny, nz, chunk)
    w = wl.small_random_case(nx=nx, ny=ny, nz=nz, pml=5, nt=12)
    with make_solver(w) as a, make_solver(w) as b:
        a.set_zchunk(chunk)
        for s in (a, b):
            s.run(0, 4)
            s.synchronize()
        before = a.field(sgfd.VX)
        a.step_phase(4, float(w.wavelet[4]), sgfd.PHASE_VELOCITY, sgfd.PART_INNER)
        a.synchronize()
        assert np.array_equal(a.field(sgfd.VX), before) != own
        a.step_phase(4, float(w.wavelet[4]), sgfd.PHASE_VELOCITY, sgfd.PART_OUTER)
        for part in (sgfd.PART_INNER, sgfd.PART_OUTER):
            a.step_phase(4, float(w.wavelet[4]), sgfd.PHASE_STRESS, part)
        for it in range(5, w.nt):
            for phase in (sgfd.PHASE_VELOCITY, sgfd.PHASE_STRESS):
                for part in (sgfd.PART_INNER, sgfd.PART_OUTER):
                    a.step_phase(it, float(w.wavelet[it]), phase, part)
        b.run(4, w.nt - 4)
        for s in (a, b):
            s.synchronize()
        np.testing.assert_array_equal(a.traces(), b.traces())
        for f in range(9):
            np.testing.assert_array_equal(a.field(f), b.field(f), err_msg=sgfd.FIELD_NAMES[f])


@pytest.mark.parametrize("nx,ny,nz", [(60, 50, 74), (234, 200, 150)])
def test_four_slabs_equal_the_whole_model(nx, ny, nz):
    w = wl.small_random_case(nx=nx, ny=ny, nz=nz, pml=5, nt=12)
    cfg = sgfd.default_config(**w.cfg)
    with sl.SlabModel(cfg, sl.plan_cuts(cfg.nz, 4, src_z=w.src[2])) as m, make_solver(w) as s:
        m.set_medium(w.b, w.lam, w.mu)
        m.set_source(*w.src)
        m.set_receivers(w.rec_xyz, w.rec_comp, w.nt)
        m.run(0, w.nt, w.wavelet)
        m.synchronize()
        s.run(0, w.nt)
        s.synchronize()
        np.testing.assert_array_equal(m.traces(), s.traces())
        for f in range(9):
            np.testing.assert_array_equal(m.field(f), s.field(f), err_msg=sgfd.FIELD_NAMES[f])
