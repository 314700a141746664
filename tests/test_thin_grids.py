"""Grids of fewer than 14 rows run on the cp.async march, whose tile is chosen for
the grid: against the direct kernel (FP64 1e-12, FP32 2e-5 per field, as
elsewhere), and the same bits with the segments of other tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DX = 0.125
TOL = {0: 1e-12, 1: 2e-5}


def solve(nb, nx, nz, nn, precision, kernel=None, tile=None):
    s = nb.NuOsc(1, 1, nn, 0, 3, 3, -nx * DX / 2, nx * DX / 2, -nz * DX / 2, nz * DX / 2, DX, DX, 0.4, 0.1,
                 precision=precision)
    assert (s.grid.nx, s.grid.nz) == (nx, nz)
    s.set_mu(1.3)
    s.set_pmo(0.2)
    if kernel is not None:
        s.set_kernel(kernel)
    if tile is not None:
        s.set_tile(*tile)
    s.fillInitValue(1, 1.2, 1e-3, 1.0, 0.6, 0.4, seed=3)
    s.step_rk4(4)
    u = s.get_state()
    s.close()
    return u


# one segment, many, the last one shorter; 4 to 13 rows; and a taller grid by name
@pytest.mark.parametrize("nx,nz,nn", [(4, 4, 1), (33, 5, 2), (512, 8, 4), (700, 13, 2), (65, 12, 5)])
@pytest.mark.parametrize("precision", [0, 1])
def test_thin(gpu, nx, nz, nn, precision):
    import nuosc_b200 as nb
    u = solve(nb, nx, nz, nn, precision)
    ref = solve(nb, nx, nz, nn, precision, nb.KERNEL_DIRECT)
    for f in range(8):
        assert np.max(np.abs(u[f] - ref[f])) <= TOL[precision] * np.max(np.abs(ref[f])), f
    for tile in ((16, 128), (8, 3)):
        assert np.array_equal(solve(nb, nx, nz, nn, precision, tile=tile), u), tile
