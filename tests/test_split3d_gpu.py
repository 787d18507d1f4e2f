"""The 3D stepping passes against the oracle, bit for bit, at the edges of their tiles.

Random states over many decades (subnormal products and quotients included)
on grids whose rows leave remainders of every size, in both precisions, for
one coefficient per cell, three per cell and the table, with and without
dispersive cells: media in 8^3 blocks (runs of cells with consecutive
records), scattered cell by cell (no runs), and with one, two and three poles.
Every operation of the passes is the reference's, rounded once, so fields
after three steps equal the oracle's exactly.
"""
import numpy as np
import pytest

import photonfdtd_b200 as pf
from photonfdtd_b200.engine import B200Engine, build_tables

pytestmark = pytest.mark.gpu

ALL6 = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")


def _box(shape, d, lo, hi, medium):
    """The cells [lo, hi) per axis."""
    c = tuple(((a + b - 1) / 2 - (n - 1) / 2) * d for a, b, n in zip(lo, hi, shape))
    return pf.Box(center=c, size=tuple((b - a) * d for a, b in zip(lo, hi)), medium=medium)


def _scene(shape, precision, media, pml, d):
    rng = np.random.default_rng(5)
    grid = pf.Grid(size=tuple(n * d for n in shape), cell_size=d, pml_layers=pml)
    dt = 0.99 * d / (pf.C_0 * 3 ** 0.5)
    u = 0.2 / dt
    pole = [pf.Pole(strength=(u * s) ** 2, omega0=u * w, gamma=u * 0.01)
            for s, w in ((1.0, 0.0), (0.5, 0.4), (0.3, 0.7))]
    mats = [pf.DispersiveMedium(eps_inf=1.0, poles=tuple(pole[:1])),
            pf.DispersiveMedium(eps_inf=2.0, poles=tuple(pole[:2])),
            pf.DispersiveMedium(eps_inf=1.5, poles=tuple(pole)),
            pf.Medium(permittivity=2.1)]
    structures = []
    if media == "blocks":
        for lo in np.ndindex(*[-(-n // 8) for n in shape]):
            m = int(rng.integers(0, 5))
            if m < 4:
                lo = [8 * v for v in lo]
                hi = [min(v + 8, n) for v, n in zip(lo, shape)]
                structures.append(_box(shape, d, lo, hi, mats[m]))
    elif media == "scattered":
        for q in range(4000):
            lo = [int(rng.integers(0, n)) for n in shape]
            structures.append(_box(shape, d, lo, [v + 1 for v in lo], mats[q % 4]))
    sim = pf.Simulation(grid, structures=structures, run_time=9.5 * dt, precision=precision)
    if media == "cell":
        sim.eps_r = rng.uniform(1.0, 12.0, size=shape).astype(precision)
    return sim


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("media", ["cell", "tensor", "blocks", "scattered"])
@pytest.mark.parametrize("shape,pml,d", [((40, 37, 64), 6, 20e-9), ((21, 70, 101), 5, 13e-9),
                                         ((18, 23, 35), (4, 0, 6), 47e-9),
                                         ((30, 9, 130), (0, 0, 0), 20e-9)])
def test_steps_bitwise_against_oracle(shape, pml, d, media, precision):
    from oracle import OracleRun
    sim = _scene(shape, precision, media, pml, d)
    rng = np.random.default_rng(7)
    ce3 = None
    if media == "tensor":
        base = sim.dt / pf.EPS_0
        ce3 = [(base * rng.uniform(0.1, 1.0, size=shape)).astype(precision) for _ in range(3)]
    lo = -40.0 if precision == "float32" else -290.0
    fields = {}
    for c in ALL6:
        mag = 10.0 ** rng.uniform(lo, 3.0, size=shape)
        fields[c] = (rng.standard_normal(shape) * mag).astype(precision)
    eng = B200Engine(build_tables(sim, ce3=ce3))
    try:
        for c in ALL6:
            eng.set_field(c, fields[c])
        eng.advance(0, 3)
        got = {c: eng.get(c).copy() for c in ALL6}
    finally:
        eng.close()
    run = OracleRun(sim, ce3=ce3)
    run.set_fields(fields)
    run.advance(3)
    for c in ALL6:
        np.testing.assert_array_equal(got[c], run.F[c], err_msg=c)
