"""nuosc_kernel_launches counts every kernel of a step and of calRHS: 4 stages and 4
moment sums, and where the tail velocities do not ride in the stage's launch (more
than 6 waves of CTAs) 4 tail kernels."""
import pytest

pytestmark = pytest.mark.gpu

DX = 0.125


def make(nb, nx, nz, nn, precision):
    s = nb.NuOsc(1, 1, nn, 0, 3, 3, -nx * DX / 2, nx * DX / 2, -nz * DX / 2, nz * DX / 2, DX, DX, 0.4, 0.1,
                 precision=precision)
    s.fillInitValue(1, 1.2, 1e-3, 1.0, 0.6, 0.4, seed=3)
    return s


# 64 x 64 cells x 162 velocities in tiles of 8 rows: per segment 8 x 2 x 6 CTAs on 2 x 148 slots
# (FP64); segments of 1 plane make 21 waves, the whole grid 1.  A last block of at most 8 (FP64) or 16
# (FP32) velocities is a tail: 162 = 5 x 32 + 2 and 644 = 10 x 64 + 4 have one, 42 = 32 + 10 and 164 =
# 2 x 64 + 36 none; 12 are
# all tail in FP32, which then has no march.
@pytest.mark.parametrize("precision,nn,lx,per_step", [(0, 4, 64, 8), (0, 4, 1, 12), (1, 8, 1, 12), (1, 4, 1, 8), (0, 2, 1, 8),
                                                      (1, 1, 1, 8)])
def test_kernels_per_step(gpu, precision, nn, lx, per_step):
    import nuosc_b200 as nb
    s = make(nb, 64, 64, nn, precision)
    s.set_tile(8, lx)
    s.step_rk4(1)
    n = nb.lib().nuosc_kernel_launches(s.handle)
    s.step_rk4(5)
    assert nb.lib().nuosc_kernel_launches(s.handle) - n == 5 * per_step
    s.close()


# 512 x 512 x 162 in FP64: at least 3 segments of 384 CTAs, 8 waves
@pytest.mark.parametrize("nx,nz,nn,kernels", [(512, 512, 4, 3), (64, 64, 4, 2), (64, 64, 2, 2)])
def test_kernels_of_calrhs(gpu, nx, nz, nn, kernels):
    import nuosc_b200 as nb
    s = make(nb, nx, nz, nn, 0)
    n = nb.lib().nuosc_kernel_launches(s.handle)
    s.calRHS(nb.REG_RHS, nb.REG_STAT)
    assert nb.lib().nuosc_kernel_launches(s.handle) - n == kernels
    s.close()
