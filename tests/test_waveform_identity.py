"""Which waveforms are evaluated for all times at once.

Only the package's own pulse and the reference's are known to be elementwise.
A user's class may carry the same name and accept one time per call, or be
derived from the pulse and look at its argument; both are called time by time,
as the reference's loop does.
"""
import sys
import types

import numpy as np
import pytest

import photonfdtd_b200 as pf
from photonfdtd_b200.engine import _elementwise, build_tables


def _user_class():
    class GaussianPulse:
        def __call__(self, t):
            if np.asarray(t).size != 1:
                raise ValueError("one time at a time")
            return np.asarray(t) * 2e15
    return GaussianPulse


class Gated(pf.GaussianPulse):
    """Derived from the pulse, with a branch on the time."""

    def __call__(self, t):
        return np.zeros(1) if t[0] < 3e-15 else super().__call__(t)


@pytest.mark.parametrize("wave", [_user_class()(), Gated(freq0=3e14, fwhm=4e-15)])
def test_user_waveforms_are_called_time_by_time(wave):
    d, steps = 20e-9, 70
    grid = pf.Grid(size=(40 * d, 40 * d), cell_size=(d, d), pml_layers=(5, 5, 0))
    dt = 0.99 * d / (pf.C_0 * 2 ** 0.5)
    src = [pf.PointDipole(position=(0, 0), component=c, waveform=wave) for c in ("Ez", "Hx")]
    t = build_tables(pf.Simulation(grid, sources=src, run_time=(steps - 0.5) * dt))
    for row, off in enumerate((1.0, 0.5)):
        want = [wave(np.array([(s + off) * t["dt"]]))[0] for s in range(steps)]
        np.testing.assert_array_equal(t["sources"]["wave"][row], want)


def test_known_pulses(monkeypatch):
    assert _elementwise(pf.GaussianPulse(freq0=3e14, fwhm=4e-15))
    ref = types.ModuleType("photonfdtd.sources")
    monkeypatch.setitem(sys.modules, "photonfdtd.sources", ref)
    exec("class GaussianPulse:\n    pass", ref.__dict__)
    assert _elementwise(ref.GaussianPulse())
    assert not _elementwise(_user_class()())
    assert not _elementwise(Gated(freq0=3e14, fwhm=4e-15))
