"""DFT monitors of an engine that is set to another step (pf_set_state).

Accumulators are not part of a state: they keep what they hold, and steps
taken again are added again. Every sample must carry the phase of its own
step, whether the engine went back or was started in the middle. The sums of
three engines are compared: one that runs through, one that goes back to step
k and runs on, one that starts at step k. All are float64 sums of the same
terms in other groupings: at most 90 roundings of 2^-53 of the largest
partial sum, which 1e-11 of the largest result covers.
"""
import numpy as np
import pytest

import photonfdtd_b200 as pf
from photonfdtd_b200.engine import B200Engine, build_tables

pytestmark = pytest.mark.gpu

COMPS = ("Ez", "Hx")


def _tables(shape, steps):
    d = 20e-9
    size = tuple(n * d if n > 1 else 0.0 for n in shape)
    grid = pf.Grid(size=size, cell_size=tuple(d if n > 1 else 0.0 for n in shape),
                   pml_layers=tuple(5 if n > 1 else 0 for n in shape))
    dt = 0.99 * d / (pf.C_0 * sum(n > 1 for n in shape) ** 0.5)
    src = pf.PointDipole(position=(0, 0, 0) if shape[2] > 1 else (0, 0), component="Ez",
                         waveform=pf.GaussianPulse(freq0=pf.C_0 / (20 * d), fwhm=9 * dt))
    mons = [pf.DFTMonitor(name="d%d" % q, components=COMPS, interval=q,
                          freqs=[pf.C_0 / (20 * d), pf.C_0 / (26 * d)]) for q in (1, 4)]
    return build_tables(pf.Simulation(grid, sources=[src], monitors=mons,
                                      run_time=(steps - 0.5) * dt, precision="float64"))


def _sums(eng, t):
    return [eng.read_dft(k, c, d["omega"].size, d["counts"])
            for k, d in enumerate(t["dft"]) for c in COMPS]


@pytest.mark.parametrize("shape", [(40, 36, 1), (24, 22, 20)])
@pytest.mark.parametrize("separate", [False, True])
@pytest.mark.parametrize("k", [0, 37, 56])
def test_phases_follow_the_step(shape, separate, k):
    steps = 90
    t = _tables(shape, steps)
    engs = [B200Engine(t) for _ in range(2)]
    try:
        for e in engs:
            e.set_profiling(separate)
        a, b = engs
        a.advance(0, k)
        blob, first = a.get_state(), _sums(a, t)
        a.advance(k, steps - k)
        whole = _sums(a, t)
        a.set_state(k, blob)
        a.advance(k, steps - k)
        twice = _sums(a, t)
        b.set_state(k, blob)
        b.advance(k, steps - k)
        rest = _sums(b, t)
    finally:
        for e in engs:
            e.close()
    for f, w, s, r in zip(first, whole, twice, rest):
        tol = 1e-11 * np.abs(w).max()
        assert tol > 0
        assert np.abs(f + r - w).max() <= tol
        assert np.abs(w + r - s).max() <= tol


@pytest.mark.parametrize("shape", [(40, 36, 1), (24, 22, 20)])
def test_phases_after_a_reverse_segment(shape):
    """A reverse segment leaves the engine at the segment's end; steps taken from
    there carry their own phases."""
    steps, n = 90, 20
    t = _tables(shape, steps)
    a, b = B200Engine(t), B200Engine(t)
    try:
        a.advance(0, steps - 2 * n)
        mid = a.get_state()
        a.advance(steps - 2 * n, n)
        last = a.get_state()
        a.advance(steps - n, n)
        a._chk(a._L.pf_adj_init(a.h, n))
        before = _sums(a, t)
        for s0, st in ((steps - n, last), (steps - 2 * n, mid)):
            a._chk(a._L.pf_adj_segment(a.h, s0, n, st.ctypes.data, st.size, 0))
        assert a.step() == steps - n
        a.advance(steps - n, n)
        after = _sums(a, t)
        b.set_state(steps - n, last)
        b.advance(steps - n, n)
        rest = _sums(b, t)
    finally:
        a.close()
        b.close()
    for x, y, r in zip(before, after, rest):
        tol = 1e-11 * np.abs(x).max()
        assert tol > 0
        assert np.abs(x + r - y).max() <= tol
