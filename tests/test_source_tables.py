"""Source waveforms and DFT phases evaluated for all times at once.

The reference evaluates them one time at a time; the tables must hold the
same bits, since the float32 parity of the stepping depends on them. A
waveform that is not the package's pulse is still called time by time.
"""
import numpy as np
import pytest

import photonfdtd_b200 as pf
from photonfdtd_b200.engine import build_tables


class Ramp:
    """A user's waveform that accepts one time per call."""

    def __call__(self, t):
        if np.asarray(t).size != 1:
            raise ValueError("one time at a time")
        return np.asarray(t) * 1e15


@pytest.mark.parametrize("steps,interval", [(1, 1), (7, 3), (64, 1), (1001, 2)])
def test_tables_equal_time_by_time_evaluation(steps, interval):
    d = 20e-9
    grid = pf.Grid(size=(40 * d, 40 * d), cell_size=(d, d), pml_layers=(5, 5, 0))
    pulse = pf.GaussianPulse(freq0=pf.C_0 / 1.1e-6, fwhm=7e-15, delay=1e-15)
    src = [pf.PointDipole(position=(0, 0), component="Ez", waveform=pulse),
           pf.PointDipole(position=(0, 0), component="Hx", waveform=pulse),
           pf.PointDipole(position=(0, 0), component="Ez", waveform=Ramp())]
    mon = pf.DFTMonitor(name="d", components=("Ez", "Hx"), interval=interval,
                        freqs=pf.C_0 / np.linspace(0.9e-6, 1.3e-6, 7))
    dt = 0.99 * d / (pf.C_0 * 2 ** 0.5)
    sim = pf.Simulation(grid, sources=src, monitors=[mon], run_time=(steps - 0.5) * dt)
    t = build_tables(sim)
    assert t["n_steps"] == steps
    dt = t["dt"]
    for row, (w, off) in enumerate([(pulse, 1.0), (pulse, 0.5), (Ramp(), 1.0)]):
        want = [w(np.array([(s + off) * dt]))[0] for s in range(steps)]
        np.testing.assert_array_equal(t["sources"]["wave"][row], want)
    om = t["dft"][0]["omega"]
    for name, off in (("ph_e", 1.0), ("ph_h", 0.5)):
        want = [np.exp(1j * om * ((s + off) * dt)) for s in range(0, steps, interval)]
        np.testing.assert_array_equal(t["dft"][0][name], np.array(want))
