"""The vector reverse step on ragged 3D grids against the oracle's transposed step.

Row lengths that leave every remainder of a vector, layers of different
widths (one axis without), both precisions, one coefficient per cell, a
table, and a loss of E and H components. The float64 gradient equals the
oracle's to 1e-10 (its own tests' bound), the float32 one to 1e-3.
"""
import numpy as np
import pytest

import photonfdtd_b200 as pf
from photonfdtd_b200.adjoint import value_and_grad_eps

pytestmark = pytest.mark.gpu


def _sim(shape, pml, precision, custom):
    d = 25e-9
    grid = pf.Grid(size=tuple(n * d for n in shape), cell_size=d, pml_layers=pml)
    dt = 0.99 * d / (pf.C_0 * 3 ** 0.5)
    box = pf.Box(center=(0.0, d, -d), size=(6 * d, 5 * d, 7 * d), medium=pf.Medium(permittivity=4.0))
    src = [pf.PointDipole(position=(0, 0, 0), component=c,
                          waveform=pf.GaussianPulse(freq0=pf.C_0 / (20 * d), fwhm=9 * dt))
           for c in ("Ex", "Hz")]
    mon = pf.DFTMonitor(name="d", components=("Ey", "Hx"), freqs=[pf.C_0 / (20 * d)],
                        plane_axis="z", plane_position=2 * d)
    sim = pf.Simulation(grid, structures=[box], sources=src, monitors=[mon],
                        run_time=39.5 * dt, precision=precision)
    if custom:
        sim.eps_r = np.random.default_rng(2).uniform(1.0, 5.0, size=shape).astype(precision)
    return sim


def _loss(out):
    return sum((v.abs() ** 2).sum() * s for v, s in zip(out["dft"]["d"].values(), (1.0, 1e5)))


@pytest.mark.parametrize("precision,tol", [("float64", 1e-10), ("float32", 1e-3)])
@pytest.mark.parametrize("shape,pml,custom", [((16, 15, 17), (4, 3, 5), False),
                                              ((13, 18, 22), (0, 4, 4), True),
                                              ((19, 12, 31), (3, 3, 0), True),
                                              ((12, 14, 36), (3, 4, 9), False)])
def test_ragged_gradient_matches_oracle(shape, pml, custom, precision, tol):
    from oracle import adjoint3d
    want_v, want = adjoint3d.value_and_grad_eps(_sim(shape, pml, "float64", custom), _loss)
    v, g = value_and_grad_eps(_sim(shape, pml, precision, custom), _loss, checkpoint_every=13)
    assert abs(v - want_v) <= tol * abs(want_v)
    err = np.linalg.norm(np.asarray(g, np.float64) - want) / np.linalg.norm(want)
    assert err <= tol, err
