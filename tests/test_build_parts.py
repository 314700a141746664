"""The build gives the same code every time: no compiler option whose result
depends on chance (--split-compile picks one of two codes), and every part of a
source compiled in parts is built (each part holds kernels of its own)."""
import importlib.util
import os
import re

from conftest import ROOT


def load_build():
    spec = importlib.util.spec_from_file_location("nuosc_build", os.path.join(ROOT, "nuosc_b200", "build.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_flags_and_parts():
    b = load_build()
    assert not [f for f in b.NVCC_FLAGS if "split-compile" in f]
    for name, n in b.PARTS.items():
        text = open(os.path.join(b.CSRC, name)).read()
        used = {int(k) for k in re.findall(r"NUOSC_PART == (\d+)", text)}
        assert used == set(range(n)), name
