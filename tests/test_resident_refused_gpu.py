"""Small grids where resident launches are refused: separate launches, the same bits.

A context may see fewer SMs than a cluster or a cooperative grid needs. The
engine asks before its first resident launch; pf_set_wait_test(2) answers no.
Launch counters tell the routes apart: separate launches are two step passes
per step. One engine is refused from the start, one after 30 steps, with
samples of the resident launches pending in its rings.
"""
import numpy as np
import pytest

import photonfdtd_b200 as pf
from photonfdtd_b200 import _native as N
from photonfdtd_b200.engine import B200Engine, build_tables

pytestmark = pytest.mark.gpu

ALL6 = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")


def _tables(shape, precision, steps):
    d = 20e-9
    size = tuple(n * d if n > 1 else 0.0 for n in shape)
    grid = pf.Grid(size=size, cell_size=tuple(d if n > 1 else 0.0 for n in shape),
                   pml_layers=tuple(4 if n > 1 else 0 for n in shape))
    dt = 0.99 * d / (pf.C_0 * sum(n > 1 for n in shape) ** 0.5)
    src = [pf.PointDipole(position=(0, 0, 0) if shape[2] > 1 else (0, 0), component=c,
                          waveform=pf.GaussianPulse(freq0=pf.C_0 / (20 * d), fwhm=9 * dt))
           for c in ("Ez", "Hx")]
    mons = [pf.DFTMonitor(name="a", components=("Ez", "Hy"), freqs=[pf.C_0 / (20 * d)], interval=3),
            pf.FluxMonitor(name="fx", plane_axis="x", plane_position=2 * d),
            pf.FluxMonitor(name="fy", plane_axis="y", plane_position=-3 * d)]
    return build_tables(pf.Simulation(grid, sources=src, monitors=mons,
                                      run_time=(steps - 0.5) * dt, precision=precision))


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("shape", [(60, 50, 1), (200, 180, 1), (500, 450, 1), (20, 30, 24)])
def test_refused_launches_fall_back(shape, precision):
    steps, turn = 77, 30
    t = _tables(shape, precision, steps)
    out = []
    for refuse_at in (None, 0, turn):
        eng = B200Engine(t)
        try:
            for at, n in ((0, turn), (turn, steps - turn)):
                if refuse_at == at:
                    N.check(N.lib().pf_set_wait_test(eng.h, 2), eng.h)
                eng.read_profile(reset=True)
                eng.advance(at, n)
                launches = eng.read_profile()[0][0]
                if refuse_at is not None and at >= refuse_at:
                    assert launches == 2 * n
                else:
                    assert launches <= n
            got = {c: eng.get(c).copy() for c in ALL6}
            got["dft"] = [eng.read_dft(0, c, 1, t["dft"][0]["counts"]) for c in ("Ez", "Hy")]
            got["flux"] = np.array([eng.read_flux(k) for k in range(2)])
        finally:
            eng.close()
        out.append(got)
    assert np.abs(out[0]["Ez"]).max() > 0 and np.abs(out[0]["flux"]).min() > 0
    for got in out[1:]:
        for k, v in out[0].items():
            np.testing.assert_array_equal(got[k], v, err_msg=str(k))
