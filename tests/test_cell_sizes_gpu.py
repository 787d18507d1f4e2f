"""Cell sizes on both sides of the reciprocal division's windows.

Infrared and terahertz grids have cells above 119 nm, atomic ones below 0.93
nm, and a grid may mix them. Quotients are IEEE quotients on all of them: the
state after a few steps from fields of all decades, subnormals included,
equals that of a run with IEEE division (PFB200_IEEE_DIV), on both routes.
"""
import numpy as np
import pytest

import photonfdtd_b200 as pf
from photonfdtd_b200.engine import B200Engine, build_tables

pytestmark = pytest.mark.gpu

ALL6 = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")


def _state(t, fields, separate, ieee, monkeypatch):
    if ieee:
        monkeypatch.setenv("PFB200_IEEE_DIV", "1")
    else:
        monkeypatch.delenv("PFB200_IEEE_DIV", raising=False)
    eng = B200Engine(t)
    try:
        eng.set_profiling(separate)
        for c in ALL6:
            eng.set_field(c, fields[c])
        eng.advance(0, 3)
        return eng.get_state().view(t["npdt"])
    finally:
        eng.close()


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("pml", [0, 5])
@pytest.mark.parametrize("cell", [(0.9e-9,) * 3, (3e-13,) * 3, (119e-9,) * 3, (121e-9,) * 3,
                                  (200e-9,) * 3, (3e-6,) * 3, (1e-3,) * 3, (20e-9, 20e-9, 200e-9),
                                  (1e-6, 0.5e-9, 130e-9)])
def test_quotients_are_ieee_quotients(cell, pml, precision, monkeypatch):
    shape = (26, 23, 38)
    grid = pf.Grid(size=tuple(n * d for n, d in zip(shape, cell)), cell_size=cell, pml_layers=pml)
    dt = 0.99 / (pf.C_0 * sum(1 / d ** 2 for d in cell) ** 0.5)
    t = build_tables(pf.Simulation(grid, run_time=9.5 * dt, precision=precision))
    rng = np.random.default_rng(6)
    lo = -45.0 if precision == "float32" else -323.0
    fields = {}
    for c in ALL6:
        # decades by block, so that some vectors hold small values alone
        dec = rng.uniform(lo, 3.0, size=tuple(-(-n // 6) for n in shape))
        dec = np.kron(dec, np.ones((6, 6, 6)))[:shape[0], :shape[1], :shape[2]]
        fields[c] = (rng.choice([-1.0, 0.0, 1.0], size=shape)
                     * 10.0 ** (dec + rng.uniform(0.0, 2.0, size=shape))).astype(precision)
    for separate in (False, True):
        got = _state(t, fields, separate, False, monkeypatch)
        want = _state(t, fields, separate, True, monkeypatch)
        assert np.count_nonzero(want) > want.size // 20
        np.testing.assert_array_equal(got, want)
