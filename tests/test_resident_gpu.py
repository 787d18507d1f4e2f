"""Small grids stepped many steps per launch against separate launches, bit for bit.

Profiling (pf_set_profiling) makes pf_advance launch every pass by itself, so
the same scene runs both ways. Grids below and above the one-cluster limit,
1D to 3D, remainders of the thread count; no source, sources of both families,
more source groups than the owner threads take; DFT monitors of several
intervals, flux on every axis, frames in between; chunks of steps that end
inside a ring.
"""
import numpy as np
import pytest

import photonfdtd_b200 as pf
from photonfdtd_b200.engine import B200Engine, build_tables

pytestmark = pytest.mark.gpu

ALL6 = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")


def _scene(shape, precision, media, n_src, steps):
    rng = np.random.default_rng(3)
    d = 20e-9
    size = tuple(n * d if n > 1 else 0.0 for n in shape)
    cell = tuple(d if n > 1 else 0.0 for n in shape)
    grid = pf.Grid(size=size, cell_size=cell, pml_layers=tuple(5 if n > 1 else 0 for n in shape))
    nd = sum(n > 1 for n in shape)
    dt = 0.99 * d / (pf.C_0 * nd ** 0.5)
    u = 0.2 / dt
    med = pf.DispersiveMedium(eps_inf=1.5, poles=(
        pf.Pole(strength=u ** 2, omega0=0.0, gamma=0.01 * u),
        pf.Pole(strength=0.5 * u ** 2, omega0=0.4 * u, gamma=0.01 * u)))
    if media == "plain":
        med = pf.Medium(permittivity=3.3)
    big = tuple(0.4 * s if s else 1e-6 for s in size)
    pulse = pf.GaussianPulse(freq0=pf.C_0 / (25 * d), fwhm=20 * dt)
    pick = lambda: tuple(float(c[rng.integers(0, len(c))]) for c in grid.coords)  # noqa: E731
    src = [pf.PointDipole(position=pick(), component=ALL6[int(rng.integers(0, 6))],
                          waveform=pulse, amplitude=1.0 + q) for q in range(n_src)]
    freqs = [pf.C_0 / (25 * d), pf.C_0 / (30 * d)]
    mons = [pf.DFTMonitor(name="a", components=("Ex", "Ez", "Hy"), freqs=freqs),
            pf.DFTMonitor(name="b", components=("Ey",), freqs=freqs, interval=3, downsample=2)]
    for ax, n in zip("xyz", shape):
        if n > 1:
            mons.append(pf.FluxMonitor(name="f" + ax, plane_axis=ax, plane_position=2.1 * d))
    return pf.Simulation(grid, structures=[pf.Box(center=(0, 0, 0), size=big, medium=med)],
                         sources=src, monitors=mons, run_time=(steps - 0.5) * dt,
                         precision=precision)


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("shape,media,n_src", [
    ((301, 1, 1), "plain", 1), ((104, 104, 1), "plain", 3), ((64, 1, 71), "ade", 40),
    ((129, 127, 1), "ade", 0), ((181, 93, 1), "ade", 2), ((13, 17, 19), "plain", 40),
    ((47, 40, 37), "ade", 3), ((411, 633, 1), "plain", 40)])
def test_resident_steps_equal_separate_launches(shape, media, n_src, precision):
    steps = 83
    t = build_tables(_scene(shape, precision, media, n_src, steps))
    out = []
    for separate in (True, False):
        eng = B200Engine(t)
        try:
            if separate:
                eng.set_profiling(True)
            pos = 0
            for n in (1, 20, 45, steps - 66):
                eng.advance(pos, n)
                pos += n
            got = {c: eng.get(c).copy() for c in ALL6}
            for k, d in enumerate(t["dft"]):
                for c in d["m"].components:
                    got[(k, c)] = eng.read_dft(k, c, d["omega"].size, d["counts"])
            for k in range(len(t["flux"])):
                got[("flux", k)] = np.array(eng.read_flux(k))
        finally:
            eng.close()
        out.append(got)
    assert n_src == 0 or any(np.abs(out[0][c]).max() > 0 for c in ALL6)
    for k, v in out[0].items():
        np.testing.assert_array_equal(v, out[1][k], err_msg=str(k))
