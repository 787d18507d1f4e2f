"""Quotients of special fields: the reciprocal division against IEEE division.

A diverging run reaches fields near the type's limits and infinities, a decayed
one subnormals, whose quotients may be subnormal themselves (float64). Every
quotient of the stepping is defined as the IEEE quotient of the difference, so
a run with the reciprocal division and one with IEEE division
(PFB200_IEEE_DIV) must hold the same state: same values, infinities and NaN in
the same places. Both routes of small grids, the vector passes included.
"""
import numpy as np
import pytest

import photonfdtd_b200 as pf
from photonfdtd_b200.batch import BatchTE
from photonfdtd_b200.engine import B200Engine, build_tables

pytestmark = pytest.mark.gpu

ALL6 = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")


def _tables(shape, pml, precision, d=20e-9):
    size = tuple(n * d if n > 1 else 0.0 for n in shape)
    grid = pf.Grid(size=size, cell_size=tuple(d if n > 1 else 0.0 for n in shape),
                   pml_layers=tuple(pml if n > 1 else 0 for n in shape))
    dt = 0.99 * d / (pf.C_0 * sum(n > 1 for n in shape) ** 0.5)
    return build_tables(pf.Simulation(grid, run_time=9.5 * dt, precision=precision))


def _state(t, fields, separate, ieee, steps, monkeypatch):
    if ieee:
        monkeypatch.setenv("PFB200_IEEE_DIV", "1")
    else:
        monkeypatch.delenv("PFB200_IEEE_DIV", raising=False)
    eng = B200Engine(t)
    try:
        eng.set_profiling(separate)
        for c in ALL6:
            eng.set_field(c, fields[c])
        eng.advance(0, steps)
        return eng.get_state().view(t["npdt"])
    finally:
        eng.close()


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("comp", ["all", "Ez", "Hz"])
@pytest.mark.parametrize("shape,pml", [((30, 26, 40), 0), ((24, 22, 37), 5), ((70, 61, 1), 4)])
def test_large_and_infinite_fields(shape, pml, comp, precision, monkeypatch):
    """Random decades with a few infinities in every component, or one component
    alone: infinite except for a few cells that overflow when prescaled, so that
    a vector of cells has no difference but infinite ones and zeros."""
    t = _tables(shape, pml, precision)
    rng = np.random.default_rng(3)
    lo, hi = (-30.0, 38.0) if precision == "float32" else (-200.0, 307.0)
    fields = {}
    for c in ALL6:
        f = rng.choice([-1.0, 1.0], size=shape) * 10.0 ** rng.uniform(lo, hi, size=shape)
        if comp == "all":
            f[rng.random(shape) < 0.02] = np.inf
            f[rng.random(shape) < 0.01] = -np.inf
        else:
            f = np.abs(f) * (c == comp)
            f[(f < 10.0 ** (0.9 * hi)) & (c == comp)] = np.inf
        fields[c] = f.astype(precision)
    for separate in (False, True):
        got = _state(t, fields, separate, False, 1, monkeypatch)
        want = _state(t, fields, separate, True, 1, monkeypatch)
        assert np.isinf(want).any() and np.isnan(want).any() and np.isfinite(want).any()
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("shape,pml", [((24, 22, 37), 5), ((31, 26, 24), 6), ((70, 61, 1), 8)])
def test_subnormal_fields(shape, pml, precision, monkeypatch):
    """The CPML state holds the quotients nearly as they are, down to the last
    subnormal bit. Float64 differences of some 2^25 units of 2^-1074 give
    subnormal quotients with one bit less than a normal one, on a cell size
    that does not divide them."""
    t = _tables(shape, pml, precision, 13e-9)
    rng = np.random.default_rng(4)
    lo, hi = (-45.0, -36.0) if precision == "float32" else (-318.0, -315.0)
    fields = {c: (rng.choice([-1.0, 0.0, 1.0], size=shape)
                  * 10.0 ** rng.uniform(lo, hi, size=shape)).astype(precision) for c in ALL6}
    for separate in (False, True):
        got = _state(t, fields, separate, False, 2, monkeypatch)
        want = _state(t, fields, separate, True, 2, monkeypatch)
        tiny = np.finfo(precision).tiny
        assert ((want != 0) & (np.abs(want) < tiny)).any()
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("precision", ["float32", "float64"])
def test_diverging_batch(precision, monkeypatch):
    d, steps = 20e-9, 24
    top = 3e38 if precision == "float32" else 1e308
    grid = pf.Grid(size=(70 * d, 66 * d), cell_size=(d, d), pml_layers=(6, 6, 0))
    dt = 0.99 * d / (pf.C_0 * 2 ** 0.5)
    pulse = pf.GaussianPulse(freq0=pf.C_0 / (20 * d), fwhm=9 * dt)
    src = [pf.PointDipole(position=(x * d, y * d), component="Ey", waveform=pulse, amplitude=a)
           for x, y, a in ((0, 0, top), (7, 3, top * 1e-9), (-9, 5, top * 1e-18))]
    mon = pf.DFTMonitor(name="out", components=("Ey",), freqs=[pf.C_0 / (20 * d)],
                        plane_axis="x", plane_position=20 * d)
    out = []
    for ieee in (False, True):
        if ieee:
            monkeypatch.setenv("PFB200_IEEE_DIV", "1")
        else:
            monkeypatch.delenv("PFB200_IEEE_DIV", raising=False)
        sim = pf.Simulation(grid, sources=src, monitors=[mon], run_time=(steps - 0.5) * dt,
                            precision=precision)
        b = BatchTE([sim], [(30, 30, 6)], tile_rows=8)
        try:
            b.forward()
            out.append([b.read_field(0, c) for c in ("Ex", "Ey", "Hz")])
        finally:
            b.close()
    assert any(np.isinf(f).any() for f in out[1]) and any(np.isnan(f).any() for f in out[1])
    for a, c in zip(*out):
        np.testing.assert_array_equal(a, c)
