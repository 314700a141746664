"""Grids that no tile height divides run on the TMA march with overlapping z
tiles, and the segment length is chosen for the grid: both against the direct
kernel (one thread per point, no tiles) at the edges of the tile geometry, with
the parity bars used elsewhere (FP64 1e-12, FP32 2e-5 per field, norm-wise).
What was refused for such grids is still refused."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DX = 0.125
TOL = {0: 1e-12, 1: 2e-5}


@pytest.fixture(scope="module")
def nb(gpu):
    import nuosc_b200
    return nuosc_b200


def make(nb, nx, nz, nn, precision, ghost, pmo=0.2):
    s = nb.NuOsc(1, 1, nn, 0, ghost, ghost, -nx * DX / 2, nx * DX / 2, -nz * DX / 2, nz * DX / 2, DX, DX, 0.4, 0.1,
                 precision=precision)
    assert (s.grid.nx, s.grid.nz) == (nx, nz)
    s.set_mu(1.3)
    s.set_pmo(pmo)
    s.fillInitValue(1, 1.2, 1e-3, 1.0, 0.6, 0.4, seed=3)
    return s


# (nx, nz): smallest x extent, 8-row tiles (14 <= nz < 22), 16-row tiles with
# the closest overlaps, one row past a multiple, long thin boxes
@pytest.mark.parametrize("nx,nz", [(4, 14), (5, 15), (7, 17), (9, 21), (4, 22), (6, 23), (13, 33), (40, 47), (3 * 16, 49),
                                   (100, 90), (5, 131)])
@pytest.mark.parametrize("precision,ghost,nn", [(0, 3, 2), (0, 2, 4), (1, 3, 4), (1, 2, 1)])
def test_ragged_against_direct(nb, nx, nz, precision, ghost, nn):
    a, b = (make(nb, nx, nz, nn, precision, ghost) for _ in range(2))
    b.set_kernel(nb.KERNEL_DIRECT)
    for s in (a, b):
        s.step_rk4(5)
    x, y = a.get_state(), b.get_state()
    for f in range(8):
        assert np.max(np.abs(x[f] - y[f])) <= TOL[precision] * np.max(np.abs(y[f])), f
    assert a.moment_error() < 1e-12
    da, db = a.analysis(), b.analysis()
    assert da["surv"] == pytest.approx(db["surv"], rel=1e-10 if precision == 0 else 2e-5)
    a.close()
    b.close()


def test_still_refused(nb):
    s = make(nb, 24, 90, 2, 0, 3)
    for call in (lambda: (s.set_kernel(nb.KERNEL_XTMA), s.step_rk4(1)), lambda: nb.Batch([s]),
                 lambda: nb._lib.check(nb.lib().nuosc_stage(s.handle, 0))):
        with pytest.raises(nb.NuoscError) as e:
            call()
        assert e.value.code == nb._lib.ERR_UNSUPPORTED
        s.set_kernel(nb.KERNEL_AUTO)
    s.close()
    p = nb._lib.Params(px=1, pz=1, nv=2, nphi=0, gx=3, gz=3, x0=-1.5, x1=1.5, z0=-1.5625, z1=1.5625, dx=DX, dz=DX,
                       cfl=0.4, ko=0.1, precision=0, device=0)
    h = C.c_void_p()
    nb._lib.check(nb.lib().nuosc_create_slab(C.byref(p), 0, C.byref(h)))  # 24 x 25 cells
    assert nb.lib().nuosc_step_rk4(h, 1) == nb._lib.ERR_UNSUPPORTED
    nb._lib.check(nb.lib().nuosc_destroy(h))
