"""The first calls of a process may come from several threads at once: each finds
the TMA kernel (asked for by name, so that any other answer is an error)."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CODE = """
import threading
import nuosc_b200 as nb
n = 8
solvers = [nb.NuOsc(1, 1, 2, 0, 3, 3, -2.0, 2.0, -2.0, 2.0, 0.125, 0.125, 0.4, 0.1) for _ in range(n)]
for s in solvers:
    s.set_kernel(nb.KERNEL_XTMA)
start, rc = threading.Barrier(n), [None] * n
def first(k):
    start.wait()
    rc[k] = nb.lib().nuosc_step_rk4(solvers[k].handle, 1)
threads = [threading.Thread(target=first, args=(k,)) for k in range(n)]
for t in threads:
    t.start()
for t in threads:
    t.join()
assert rc == [0] * n, rc
"""


@pytest.mark.parametrize("attempt", range(3))
def test_first_step_from_many_threads(gpu, attempt):
    r = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
