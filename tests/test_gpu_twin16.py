"""The two-planes-at-a-time kernels of 16-bit storage where they can go wrong:
chunks of one plane, odd chunks and odd heights (a pair with one plane), rows
and columns past the last tile, borders of every width down to one cell and
none, every damping profile and quirk mode: bit-exact against the oracle's
emulation, scale changes included."""
import numpy as np
import pytest

from helpers import make_solver, run_oracle
import sgfd
import sgfd.workloads as wl

pytestmark = pytest.mark.gpu

# nx, ny, nz, pml, z chunk, quirks, damping
CASES = [
    (23, 21, 22, 1, 1, sgfd.QUIRKS_REF, sgfd.DAMP_LOGR),
    (43, 19, 21, 2, 2, sgfd.QUIRKS_FIXED, sgfd.DAMP_REFCPU),
    (75, 27, 24, 5, 3, sgfd.QUIRKS_REF, sgfd.DAMP_REFGPU),
    (42, 34, 31, 8, 5, sgfd.QUIRKS_FIXED, sgfd.DAMP_LOGR),
    (74, 58, 33, 6, 23, sgfd.QUIRKS_FIXED, sgfd.DAMP_LOGR),
    (38, 30, 25, 0, 4, sgfd.QUIRKS_REF, sgfd.DAMP_LOGR),
]


@pytest.mark.parametrize("storage", [sgfd.STORE_BF16, sgfd.STORE_F16], ids=["bf16", "f16"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "%dx%dx%d_pml%d_chunk%d" % c[:5])
def test_tile_and_pair_edges(case, storage):
    nx, ny, nz, pml, chunk, quirks, damping = case
    w = wl.small_random_case(nx=nx, ny=ny, nz=nz, pml=max(pml, 1), nt=20, quirks=quirks, damping=damping)
    w.cfg["pml"] = pml
    w.cfg["storage"] = storage
    o = run_oracle(w)
    with make_solver(w) as s:
        s.set_zchunk(chunk)
        s.run(0, w.nt, graph=False)
        s.synchronize()
        np.testing.assert_array_equal(s.traces(), o.traces().astype(np.float32))
        for fid in range(9):
            np.testing.assert_array_equal(s.field(fid), o.field(fid).astype(np.float32),
                                          err_msg=sgfd.FIELD_NAMES[fid])
