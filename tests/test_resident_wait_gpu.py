"""The grid barrier of resident launches is bounded.

With the test hook every block waits for arrivals that never come and gives up
after a few milliseconds, the kernel ends, and pf_advance reports
PF_ERR_TIMEOUT. The next engine is right: the context survived.
"""
import numpy as np
import pytest

import photonfdtd_b200 as pf
from photonfdtd_b200 import _native as N
from photonfdtd_b200.engine import B200Engine, build_tables

pytestmark = pytest.mark.gpu


def _tables(n, precision):
    d = 20e-9
    grid = pf.Grid(size=(n * d, n * d), cell_size=(d, d), pml_layers=(5, 5, 0))
    dt = 0.99 * d / (pf.C_0 * 2 ** 0.5)
    src = pf.PointDipole(position=(0, 0), component="Ez",
                         waveform=pf.GaussianPulse(freq0=pf.C_0 / (20 * d), fwhm=9 * dt))
    return build_tables(pf.Simulation(grid, sources=[src], run_time=39.5 * dt,
                                      precision=precision))


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("n", [150, 601])  # one cell per thread, several
def test_grid_barrier_runs_out_and_is_reported(n, precision):
    t = _tables(n, precision)

    def run(hook):
        eng = B200Engine(t)
        try:
            N.check(N.lib().pf_set_wait_test(eng.h, hook), eng.h)
            eng.advance(0, 40)
            return eng.get("Ez").copy()
        finally:
            eng.close()
    a = run(0)
    with pytest.raises(N.NativeError) as ei:
        run(1)
    assert ei.value.code == N.PF_ERR_TIMEOUT
    assert "grid barrier" in str(ei.value)
    np.testing.assert_array_equal(run(0), a)
    np.testing.assert_array_equal(run(2), a)
