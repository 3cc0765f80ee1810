"""16-bit storage with a NaN in one cell: on a scale-choosing step the field's
largest written magnitude is then not finite and its exponent stays, whichever
cell of a pair (planes of the 32 x 8 kernels, columns of the 64 x 8 kernels)
holds the NaN.  The z-marching kernels' fields equal the per-cell kernels' bit
for bit."""
import numpy as np
import pytest

from helpers import make_solver
import sgfd
import sgfd.workloads as wl

pytestmark = pytest.mark.gpu


def fields(x, z, storage, kernel, tile):
    """All fields after step 0 and after step 1, lambda NaN at one interior cell
    whose tile holds no PML cell."""
    w = wl.small_random_case(nx=111, ny=41, nz=45, pml=5, nt=4, quirks=sgfd.QUIRKS_FIXED, damping=sgfd.DAMP_LOGR)
    w.lam = w.lam.copy()
    w.lam[z, 20, x] = np.nan
    w.src = (50, 20, 22)
    w.wavelet = w.wavelet + np.float32(1e9)
    out = []
    with make_solver(w, storage=storage, kernel=kernel) as s:
        if tile:
            s.set_tile(*tile)
        for it in (0, 1):
            s.run(it, 1, graph=False)
            s.synchronize()
            out += [s.field(f).view(np.uint32) for f in range(9)]
    return out


@pytest.mark.parametrize("storage", [sgfd.STORE_BF16, sgfd.STORE_F16], ids=["bf16", "f16"])
@pytest.mark.parametrize("x,z", [(50, 20), (51, 21)])
@pytest.mark.parametrize("tile", [(32, 8, 8), (32, 8, 7), (64, 8, 8)], ids=lambda t: "%dx%d_chunk%d" % t)
def test_nan_keeps_the_exponents(tile, x, z, storage):
    want = fields(x, z, storage, sgfd.KERNEL_SIMPLE, None)
    got = fields(x, z, storage, sgfd.KERNEL_AUTO, tile)
    for k, (a, b) in enumerate(zip(got, want)):
        np.testing.assert_array_equal(a, b, err_msg="step %d, %s" % (k // 9, sgfd.FIELD_NAMES[k % 9]))
