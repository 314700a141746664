"""Which kernel calRHS takes: the TMA march, or the direct kernel for the smallest
4th-difference calls (fewer than 40,000 values a field).  Asked for by name the
march runs there too, and agrees with the direct kernel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DX = 0.125
TOL = {0: 1e-13, 1: 2e-6}  # of each field's maximum, as elsewhere for calRHS


# points per field: 5,376 and 38,808 (direct at ghost 2), 40,320 (march), 12 velocities
@pytest.mark.parametrize("nx,nz,nn", [(8, 16, 2), (21, 44, 2), (20, 48, 2), (4, 14, 1), (5, 17, 3), (9, 33, 2)])
@pytest.mark.parametrize("precision,ghost", [(0, 2), (1, 2), (0, 3), (1, 3)])
def test_route(gpu, nx, nz, nn, precision, ghost):
    import nuosc_b200 as nb
    s = nb.NuOsc(1, 1, nn, 0, ghost, ghost, -nx * DX / 2, nx * DX / 2, -nz * DX / 2, nz * DX / 2, DX, DX, 0.4, 0.1,
                 precision=precision)
    s.set_mu(1.3)
    s.set_pmo(0.4)
    s.set_state(np.random.default_rng(7).uniform(-1.0, 1.0, size=(8, nx, nz, s.grid.nv)))
    out = {}
    for kind in (nb.KERNEL_AUTO, nb.KERNEL_XTMA, nb.KERNEL_DIRECT):
        s.set_kernel(kind)
        s.calRHS(nb.REG_RHS, nb.REG_STAT)
        out[kind] = s.get_state(nb.REG_RHS)
    ref = out[nb.KERNEL_DIRECT]
    for f in range(8):
        assert np.max(np.abs(out[nb.KERNEL_XTMA][f] - ref[f])) <= TOL[precision] * np.max(np.abs(ref[f])), f
    march = ghost == 3 or nx * nz * s.grid.nv_stride >= 40000
    s.close()
    assert np.array_equal(out[nb.KERNEL_AUTO], out[nb.KERNEL_XTMA if march else nb.KERNEL_DIRECT])
