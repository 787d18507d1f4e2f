"""Engines before and after cudaDeviceReset in one process.

The library keeps a memory pool and pinned error words from one engine to the
next; a reset destroys both. An engine built afterwards must get its own, and
give the same bits. Run in a child process: the reset ends the process's
whole context.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes, glob, os, sys
import numpy as np
import photonfdtd_b200 as pf
from photonfdtd_b200.engine import B200Engine, build_tables

d = 20e-9
grid = pf.Grid(size=(60 * d, 50 * d), cell_size=(d, d), pml_layers=(5, 5, 0))
dt = 0.99 * d / (pf.C_0 * 2 ** 0.5)
src = pf.PointDipole(position=(0, 0), component="Ez",
                     waveform=pf.GaussianPulse(freq0=pf.C_0 / (20 * d), fwhm=9 * dt))
t = build_tables(pf.Simulation(grid, sources=[src], run_time=39.5 * dt))


def run():
    eng = B200Engine(t)
    try:
        eng.advance(0, 40)
        return eng.get("Ez").copy()
    finally:
        eng.close()


a = run()
assert np.abs(a).max() > 0
import torch
base = os.path.dirname(os.path.dirname(torch.__file__))
path = glob.glob(os.path.join(base, "nvidia", "cuda_runtime", "lib", "libcudart.so*"))
rt = ctypes.CDLL(path[0] if path else "libcudart.so.12")
for _ in range(2):
    assert rt.cudaDeviceReset() == 0
    for _ in range(3):
        np.testing.assert_array_equal(run(), a)
print("ok")
"""


def test_engines_after_a_device_reset():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD], cwd=root, timeout=300, capture_output=True,
                       text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
