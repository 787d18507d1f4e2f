"""The batch's vector steps against its split passes, bit for bit, at the edges of their tiles.

Instances whose bulk region is empty, one tile, or leaves remainders of rows
and columns; layers of several widths; design windows and output lines inside
the bulk and in the frame; Ex and Ey sources, several on one cell, and on the
output line itself. Forward DFT, fields and the design gradient of the two
forms must be equal (PFB200_BATCH_SPLIT=1 selects the split passes).
"""
import numpy as np
import pytest

import photonfdtd_b200 as pf
from photonfdtd_b200.batch import BatchTE

pytestmark = pytest.mark.gpu

SHAPES = [(40, 36), (61, 77), (64, 96), (83, 129), (50, 160), (131, 66), (33, 33)]


def _sims(precision, pml, steps):
    rng = np.random.default_rng(11)
    d = 20e-9
    sims, windows = [], []
    for k, (nx, ny) in enumerate(SHAPES):
        grid = pf.Grid(size=(nx * d, ny * d), cell_size=(d, d), pml_layers=(pml, pml, 0))
        xs, ys = grid.coords[0], grid.coords[1]
        dt = 0.99 * d / (pf.C_0 * 2 ** 0.5)
        pulse = pf.GaussianPulse(freq0=pf.C_0 / 1.0e-6, fwhm=12 * dt)
        line = int(rng.integers(2, nx - 2))
        src = []
        for q in range(9):
            i = line if q == 0 else int(rng.integers(1, nx - 1))
            j = int(rng.integers(1, ny - 1))
            for _ in range(2 if q == 1 else 1):
                src.append(pf.PointDipole(position=(float(xs[i]), float(ys[j])),
                                          component=("Ey", "Ex")[q % 2], waveform=pulse,
                                          amplitude=1.0 + 0.1 * q))
        mon = pf.DFTMonitor(name="out", components=("Ey",), freqs=pf.C_0 / np.linspace(0.8e-6, 1.2e-6, 3),
                            plane_axis="x", plane_position=float(xs[line]))
        sim = pf.Simulation(grid, sources=src, monitors=[mon], run_time=(steps - 0.5) * dt,
                            precision=precision)
        sim.eps_r = rng.uniform(1.0, 9.0, size=(nx, ny, 1)).astype(precision)
        n = int(rng.integers(3, 24))
        sims.append(sim)
        windows.append((int(rng.integers(0, nx - n)), int(rng.integers(0, ny - n)), n))
    return sims, windows


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("pml,tile_rows", [(0, 8), (5, 8), (8, 16), (12, 32), (3, 32)])
def test_vector_steps_equal_split_passes(pml, tile_rows, precision, monkeypatch):
    steps = 70
    sims, windows = _sims(precision, pml, steps)
    out = []
    for split in (False, True):
        if split:
            monkeypatch.setenv("PFB200_BATCH_SPLIT", "1")
        else:
            monkeypatch.delenv("PFB200_BATCH_SPLIT", raising=False)
        b = BatchTE(sims, windows, tile_rows=tile_rows, checkpoint_every=29)
        try:
            F = b.forward()
            got = [F] + [b.read_field(k, c) for k in range(len(sims)) for c in ("Ex", "Ey", "Hz")]
            got.append(b.adjoint(F))
        finally:
            b.close()
        out.append(got)
    assert np.abs(out[0][0]).max() > 0 and np.abs(out[0][-1]).max() > 0
    for a, c in zip(*out):
        np.testing.assert_array_equal(a, c)
