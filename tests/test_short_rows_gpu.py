"""Grids of a few cells along z: what their rows take, and their bits.

Short rows are padded to 16 bytes, so a grid of four float cells along z holds
no more than its cells; the steps equal the oracle's on every short length,
CPML along x and y, on both routes.
"""
import numpy as np
import pytest

import photonfdtd_b200 as pf
from photonfdtd_b200.engine import B200Engine, build_tables

pytestmark = pytest.mark.gpu

ALL6 = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")


def _sim(shape, precision):
    d = 20e-9
    grid = pf.Grid(size=tuple(n * d for n in shape), cell_size=d, pml_layers=(4, 4, 0))
    dt = 0.99 * d / (pf.C_0 * 3 ** 0.5)
    sim = pf.Simulation(grid, run_time=9.5 * dt, precision=precision)
    sim.eps_r = np.random.default_rng(2).uniform(1.0, 9.0, size=shape).astype(precision)
    return sim


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("nz", [4, 5, 8, 9, 12, 15, 16, 17, 31, 32, 33])
def test_short_rows_bitwise_against_oracle(nz, precision):
    from oracle import OracleRun
    shape = (21, 18, nz)
    sim = _sim(shape, precision)
    rng = np.random.default_rng(4)
    fields = {c: rng.standard_normal(shape).astype(precision) for c in ALL6}
    run = OracleRun(sim)
    run.set_fields(fields)
    run.advance(3)
    t = build_tables(sim)
    for separate in (True, False):
        eng = B200Engine(t)
        try:
            eng.set_profiling(separate)
            for c in ALL6:
                eng.set_field(c, fields[c])
            eng.advance(0, 3)
            for c in ALL6:
                np.testing.assert_array_equal(eng.get(c), run.F[c], err_msg=c)
        finally:
            eng.close()


def test_four_cells_along_z_take_no_padding():
    shape = (600, 500, 4)
    eng = B200Engine(build_tables(_sim(shape, "float32")))
    try:
        # six fields and one coefficient, then the x and y layers' state
        cells = int(np.prod(shape))
        layers = 12 * 4 * 8 * max(shape[0], shape[1]) * 4
        assert eng.device_bytes() <= 4 * (7 * cells + layers) + (2 << 20)
    finally:
        eng.close()
