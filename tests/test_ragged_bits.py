"""Grids that no tile height divides are repeatable bit for bit: every row of
the state and of the moment partials is stored by one tile, so no result
depends on which of two overlapping tiles comes last, and a solve continued
from a checkpoint equals the uninterrupted one.  Nor does a result depend on the
tile's height or on where in a tile a row lies."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DX = 0.125


@pytest.fixture(scope="module")
def nb(gpu):
    import nuosc_b200
    return nuosc_b200


def make(nb, nx, nz, nn, precision, ghost, tile=None):
    s = nb.NuOsc(1, 1, nn, 0, ghost, ghost, -nx * DX / 2, nx * DX / 2, -nz * DX / 2, nz * DX / 2, DX, DX, 0.4, 0.1,
                 precision=precision)
    assert (s.grid.nx, s.grid.nz) == (nx, nz)
    s.set_mu(1.3)
    s.set_pmo(0.2)
    if tile:
        s.set_tile(*tile)
    s.fillInitValue(1, 1.2, 0.1, 1.0, 0.6, 0.4, seed=3)
    return s


def bits(s):
    return s.get_state().view(np.uint64)


# tiles that start at odd distances from each other, by one row and by many
@pytest.mark.parametrize("nz", [17, 22, 33, 49, 90, 150])
@pytest.mark.parametrize("precision,ghost,nn", [(0, 3, 4), (1, 2, 4)])
def test_repeatable(nb, nz, precision, ghost, nn, tmp_path):
    ref = None
    for _ in range(5):
        s = make(nb, 64, nz, nn, precision, ghost)
        s.step_rk4(12)
        ref = bits(s) if ref is None else ref
        assert np.array_equal(bits(s), ref)
        s.close()
    a = make(nb, 64, nz, nn, precision, ghost)
    a.step_rk4(5)
    path = str(tmp_path / "ck.bin")
    a.save_checkpoint(path)
    a.close()
    b = make(nb, 64, nz, nn, precision, ghost)
    b.load_checkpoint(path)
    b.step_rk4(7)
    assert np.array_equal(bits(b), ref)
    b.close()


# 8- and 16-row tiles put a row at an odd place in one tile and at an even one in
# the other; segments of one and of many planes
@pytest.mark.parametrize("nz", [22, 33, 49, 90, 150])
@pytest.mark.parametrize("precision,ghost,nn", [(0, 3, 4), (0, 2, 3), (1, 3, 3), (1, 2, 4)])
def test_tile_independent(nb, nz, precision, ghost, nn):
    ref = None
    for tile in ((16, 128), (8, 128), (16, 3), (8, 5)):
        s = make(nb, 24, nz, nn, precision, ghost, tile)
        s.step_rk4(5)
        ref = bits(s) if ref is None else ref
        assert np.array_equal(bits(s), ref), tile
        s.close()
