"""The diagnostics' reduction over rows of any length: rows of three 16-byte vectors
(12 velocities in FP32), rows with padding, more and fewer rows than the device's
threads take at a time, against numpy on the state that it reads."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DX = 0.125


@pytest.mark.parametrize("nx,nz,nn", [(4, 4, 1), (5, 7, 5), (4, 14, 20), (300, 100, 1), (64, 70, 2), (33, 40, 8)])
@pytest.mark.parametrize("precision", [0, 1])
def test_against_numpy(gpu, nx, nz, nn, precision):
    import nuosc_b200 as nb
    s = nb.NuOsc(1, 1, nn, 0, 3, 3, -nx * DX / 2, nx * DX / 2, -nz * DX / 2, nz * DX / 2, DX, DX, 0.4, 0.1,
                 precision=precision)
    assert (s.grid.nx, s.grid.nz) == (nx, nz)
    s.fillInitValue(1, 1.2, 0.1, 1.0, 0.6, 0.4, seed=3)
    u = s.get_state()
    # the spectra, from the cell of the initial data itself (ee + mm is G, in FP32 to 1e-7)
    g, gb = u[0, 0, 0] + u[1, 0, 0], u[4, 0, 0] + u[5, 0, 0]
    s.step_rk4(3)
    u, d, w = s.get_state(), s.analysis(), s.grid.vw
    s.close()
    cells = nx * nz
    sums = {"surv": np.sum(u[0] * w) / np.sum(g * w) / cells, "survb": np.sum(u[4] * w) / np.sum(gb * w) / cells,
            "aM0": np.sqrt(np.sum((u[2] - u[6]) * w) ** 2 + np.sum((u[3] + u[7]) * w) ** 2 +
                           (0.5 * np.sum((u[0] - u[1] - u[4] + u[5]) * w)) ** 2) / cells}
    length = np.sqrt(4 * u[2] ** 2 + 4 * u[3] ** 2 + (u[0] - u[1]) ** 2) / g
    lengthb = np.sqrt(4 * u[6] ** 2 + 4 * u[7] ** 2 + (u[4] - u[5]) ** 2) / gb
    tol = 1e-12 if precision == 0 else 1e-6  # (FP32: the spectra as this test has them)
    for k, x in sums.items():
        assert d[k] == pytest.approx(x, rel=tol), k
    assert d["maxdP"] == pytest.approx(max(np.max(np.abs(1 - length)), np.max(np.abs(1 - lengthb))), abs=tol)
    assert d["avgP"] == pytest.approx(np.sum(w * g * np.abs(1 - length)) / np.sum(w * g) / cells, abs=tol)
