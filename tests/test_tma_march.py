"""The TMA march kernel gives the same bits for every tile shape, alone and in
a batch: each point sees the same operations in the same order whatever tile
it falls into, so any difference is a value read too early or too late.
Segments shorter than the ghost width, ragged last segments and more CTAs than
the device holds at once (rings refilled under contention) are included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DX = 0.125


@pytest.fixture(scope="module")
def nb(gpu):
    import nuosc_b200
    return nuosc_b200


def solve(nb, nx, nz, nn, precision, ghost, tile, steps, batch=False, pmo=0.0):
    s = nb.NuOsc(1, 1, nn, 0, ghost, ghost, -nx * DX / 2, nx * DX / 2, -nz * DX / 2, nz * DX / 2, DX, DX, 0.4, 0.1,
                 precision=precision)
    s.set_mu(1.0)
    s.set_pmo(pmo)
    s.set_tile(*tile)
    s.set_kernel(nb.KERNEL_XTMA)
    s.fillInitValue(1, 0.9, 0.1, 0.6, 0.6, 0.5, seed=23)
    if batch:
        with nb.Batch([s]) as b:
            b.step_rk4(steps)
            b.synchronize()
    else:
        s.step_rk4(steps)
        s.synchronize()
    st = s.get_state().view(np.uint64)
    s.close()
    return st


@pytest.mark.parametrize("pmo", [0.0, 0.3])
@pytest.mark.parametrize("ghost", [3, 2])
@pytest.mark.parametrize("precision", [0, 1])
def test_tiles_bit_identical(nb, precision, ghost, pmo):
    ref = None
    for tile in ((16, 128), (16, 1), (16, 2), (8, 5), (8, 7), (8, 1), (16, 16)):
        for batch in (False, True):
            st = solve(nb, 33, 32, 4, precision, ghost, tile, 3, batch, pmo)
            ref = st if ref is None else ref
            assert np.array_equal(st, ref), (tile, batch)


@pytest.mark.parametrize("precision", [0, 1])
def test_many_short_tiles_repeatable(nb, precision):
    """1280 CTAs of 16 planes, two per SM: five runs equal the run with whole-length segments."""
    ref = solve(nb, 128, 128, 4, precision, 3, (16, 128), 4)
    for _ in range(5):
        assert np.array_equal(solve(nb, 128, 128, 4, precision, 3, (8, 16), 4), ref)
