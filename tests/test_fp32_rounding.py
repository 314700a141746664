"""The FP32 march sums the stencil without rounding at more than its terms' size: a
uniform state without self-interaction is kept.  Its stencil sums are zero but for
rounding, the same in every cell and step, so that an error that reaches the state's
last bit grows with the steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DX = 0.125


# One ulp of a value U is what the step's last stage may be off by: B = U + Y2 + dt k2 is
# rounded at 2 U (half of 2 ulp), B + Y4 at 3 U (half of 4 ulp), and a third of the two is 1.
# With all 13 terms of the stencil in one chain the values drift by 2.
@pytest.mark.parametrize("ghost", [2, 3])
@pytest.mark.parametrize("nn", [4, 8])
def test_uniform_state_is_kept(gpu, ghost, nn):
    import nuosc_b200 as nb
    s = nb.NuOsc(1, 1, nn, 0, ghost, ghost, -2.0, 2.0, -2.0, 2.0, DX, DX, 0.4, 0.1, precision=nb.FP32)
    s.set_mu(0.0)
    s.set_pmo(0.0)
    u = np.empty((8, 32, 32, s.grid.nv))
    u[:] = np.random.default_rng(3).uniform(0.5, 1.0, size=(8, 1, 1, s.grid.nv)).astype(np.float32)
    s.set_state(u)
    s.step_rk4(60)
    err = np.abs(s.get_state() - u) / np.spacing(u.astype(np.float32))
    s.close()
    assert err.max() <= 1.0
