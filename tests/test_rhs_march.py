"""calRHS on the TMA march against the direct kernel, through the handle and on
a caller's own buffers, at the edges of the tile geometry (the calRHS bar used
elsewhere: 1e-13 of each field's maximum in FP64; 2e-6 in FP32, some tens of
float roundings of sums of 13 terms), and buffers the march cannot take."""
import ctypes as C

import numpy as np
import pytest

from test_zz_no_alloc import RhsDesc

pytestmark = pytest.mark.gpu

DX = 0.125
TOL = {0: 1e-13, 1: 2e-6}


def close(got, ref, tol):
    return all(np.max(np.abs(got[f] - ref[f])) <= tol * np.max(np.abs(ref[f])) for f in range(8))


@pytest.mark.parametrize("nx,nz", [(4, 14), (5, 17), (4, 22), (9, 33), (40, 48), (23, 90)])
@pytest.mark.parametrize("precision,ghost,nn", [(0, 3, 4), (0, 2, 2), (1, 3, 3), (1, 2, 8)])
def test_calrhs_march_against_direct(gpu, nx, nz, precision, ghost, nn):
    import torch
    import nuosc_b200 as nb
    s = nb.NuOsc(1, 1, nn, 0, ghost, ghost, -nx * DX / 2, nx * DX / 2, -nz * DX / 2, nz * DX / 2, DX, DX, 0.4, 0.1,
                 precision=precision)
    s.set_mu(1.3)
    s.set_pmo(0.4)
    g = s.grid
    state = np.random.default_rng(5).uniform(-1.0, 1.0, size=(8, nx, nz, g.nv))
    s.set_state(state)
    s.calRHS(nb.REG_RHS, nb.REG_STAT)
    got = s.get_state(nb.REG_RHS)
    s.set_kernel(nb.KERNEL_DIRECT)
    s.calRHS(nb.REG_PRE, nb.REG_STAT)
    ref = s.get_state(nb.REG_PRE)
    assert close(got, ref, TOL[precision])
    # the caller's buffers: aligned rows (the march), rows or a base that are not
    # 16-byte aligned (the direct kernel)
    dev = torch.device("cuda", 0)
    dtype = torch.float64 if precision == nb.FP64 else torch.float32
    fn = nb.lib().nuosc_calrhs_noalloc
    fn.argtypes = [C.POINTER(RhsDesc), C.c_void_p, C.c_void_p, C.c_void_p]
    fn.restype = C.c_int
    for stride, shift in ((g.nv_stride, 0), (g.nv_stride + 1, 0), (g.nv_stride, 1)):
        quad = []
        for a in (g.vx, g.vy, g.vz, g.vw):
            t = torch.zeros(stride, dtype=torch.float64, device=dev)
            t[:g.nv] = torch.tensor(a, device=dev)
            quad.append(t)
        n = 8 * nx * nz * stride
        src, dst = (torch.zeros(n + 1, dtype=dtype, device=dev) for _ in range(2))
        src[shift:shift + n].view(8, nx, nz, stride)[..., :g.nv] = torch.tensor(state, device=dev).to(dtype)
        desc = RhsDesc(nx=nx, nz=nz, nv=g.nv, nv_stride=stride, precision=precision, ko_order=6 if ghost == 3 else 4,
                       dx=DX, dz=DX, ko=0.1, mu=1.3, pmo=0.4, vx=quad[0].data_ptr(), vy=quad[1].data_ptr(),
                       vz=quad[2].data_ptr(), vw=quad[3].data_ptr())
        size = src.element_size()
        rc = fn(C.byref(desc), src.data_ptr() + shift * size, dst.data_ptr() + shift * size,
                torch.cuda.current_stream(dev).cuda_stream)
        assert rc == 0, nb.lib().nuosc_last_error()
        torch.cuda.synchronize(dev)
        out = dst[shift:shift + n].view(8, nx, nz, stride).double().cpu().numpy()[..., :g.nv]
        assert close(out, ref, TOL[precision]), (stride, shift)
    s.close()
