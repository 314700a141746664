"""The z tiles of the TMA kernels, on the host arithmetic that the launches use
(no GPU): every tile lies inside the grid, whatever its size, and every row is
stored by one tile."""
import ctypes as C

import pytest

from nuosc_b200 import _lib


def z_tile(lib, nz, tz, tile):
    z0, skip = C.c_int(), C.c_int()
    _lib.check(lib.nuosc_selftest_z_tile(nz, tz, tile, C.byref(z0), C.byref(skip)))
    return z0.value, skip.value


@pytest.fixture(scope="module")
def lib():
    import nuosc_b200
    return nuosc_b200.lib()


def rows_of(lib, nz, tz):
    return [z_tile(lib, nz, tz, t) for t in range(-(-nz // tz))]


# around every multiple of both heights, and around the sizes from which the
# product tile x (nz - tz) leaves 32 bits (131,080 and 185,377), up to the
# 65,535 tiles that a launch can have
@pytest.mark.parametrize("tz", [8, 16])
def test_starts(lib, tz):
    for nz in [*range(tz + 6, 200), 131079, 131080, 131081, 185376, 185377, 185392, 262144, 524272, 65535 * tz]:
        if -(-nz // tz) > 65535:
            continue
        n = -(-nz // tz)
        starts, skip = zip(*rows_of(lib, nz, tz))
        assert list(starts) == [t * (nz - tz) // (n - 1) for t in range(n)]
        assert starts[0] == 0 and starts[-1] == nz - tz
        if nz % tz == 0:
            assert list(starts) == list(range(0, nz, tz)) and not any(skip)
        # no gap, and at least as far apart as the widest halo (3 rows)
        assert all(3 <= b - a <= tz for a, b in zip(starts, starts[1:]))
        # the rows that the tiles store follow each other and are all of the grid's
        assert [a + k for a, k in zip(starts, skip)] == [0] + [a + tz for a in starts[:-1]]


def test_no_such_tile(lib):
    for nz, tz, tile in ((90, 12, 0), (21, 16, 0), (90, 16, 6), (90, 16, -1), (65535 * 16 + 1, 16, 0)):
        assert lib.nuosc_selftest_z_tile(nz, tz, tile, None, None) == _lib.ERR_INVALID
