"""Very tall grids: rows beyond 185,377, where a product of tile and rows leaves 32
bits, against the direct kernel; and more rows than a TMA launch has tiles for
(65,535 of 16), which other kernels run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DX = 0.125


def make(nb, nz):
    s = nb.NuOsc(1, 1, 1, 0, 3, 3, -2 * DX, 2 * DX, -nz * DX / 2, nz * DX / 2, DX, DX, 0.4, 0.1)
    assert (s.grid.nx, s.grid.nz) == (4, nz)
    s.set_mu(1.3)
    s.set_pmo(0.2)
    s.fillInitValue(1, 1.2, 1e-3, 1.0, 0.6, 0.4, seed=3)
    return s


# no tile height divides the first; 8-row tiles of the second
@pytest.mark.parametrize("nz", [185393, 185400])
def test_rows_beyond_32_bit_products(gpu, nz):
    import nuosc_b200 as nb
    out = []
    for kind in (nb.KERNEL_AUTO, nb.KERNEL_DIRECT):
        s = make(nb, nz)
        s.set_kernel(kind)
        s.step_rk4(2)
        out.append(s.get_state())
        s.calRHS(nb.REG_RHS, nb.REG_STAT)
        out.append(s.get_state(nb.REG_RHS))
        s.close()
    for f in range(8):
        assert np.max(np.abs(out[0][f] - out[2][f])) <= 1e-12 * np.max(np.abs(out[2][f])), f
        # (calRHS of states that differ by that: its weights are below 1e2)
        assert np.max(np.abs(out[1][f] - out[3][f])) <= 1e-10 * np.max(np.abs(out[2])), f


def test_more_rows_than_tiles(gpu):
    import nuosc_b200 as nb
    nz = 65535 * 16 + 2
    diag = []
    for kind in (nb.KERNEL_AUTO, nb.KERNEL_XMARCH):
        s = make(nb, nz)
        s.set_kernel(kind)
        s.step_rk4(1)
        s.calRHS(nb.REG_RHS, nb.REG_STAT)
        diag.append(s.analysis())
        s.close()
    assert diag[0] == diag[1]
