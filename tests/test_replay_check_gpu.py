"""The periodic finite check during a reverse segment's replay.

The vector passes write a replay's H into the step's record, not into the
engine's own arrays; the check must look there. An H source on the grid's
first plane overflows float32: no E update reads that H cell, so H alone
becomes infinite. The vector passes (3D) and the scalar ones.
"""
import numpy as np
import pytest

import photonfdtd_b200 as pf
from photonfdtd_b200 import _native as N
from photonfdtd_b200.engine import B200Engine, build_tables

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(20, 18, 24), (90, 88, 93), (40, 36, 1)])
def test_replay_stops_at_the_first_infinite_h(shape):
    d, n, at = 20e-9, 12, 8
    size = tuple(m * d if m > 1 else 0.0 for m in shape)
    grid = pf.Grid(size=size, cell_size=tuple(d if m > 1 else 0.0 for m in shape), pml_layers=0)
    dt = 0.99 * d / (pf.C_0 * sum(m > 1 for m in shape) ** 0.5)

    def wave(t):
        return np.where(t > (at + 0.1) * dt, 1e39, 0.0)
    pos = [float(grid.coords[a][0 if a == 0 else shape[a] // 2]) for a in range(3) if shape[a] > 1]
    src = pf.PointDipole(position=tuple(pos), component="Hx", waveform=wave)
    t = build_tables(pf.Simulation(grid, sources=[src], run_time=(n - 0.5) * dt,
                                   precision="float32"))
    eng = B200Engine(t)
    try:
        blob = eng.get_state()
        eng.advance(0, n)
        assert all(np.isfinite(eng.get(c)).all() for c in ("Ex", "Ey", "Ez", "Hy", "Hz"))
        assert np.isinf(eng.get("Hx")).any()
        eng._chk(eng._L.pf_adj_init(eng.h, n))
        eng.set_check_every(1)
        with pytest.raises(N.NativeError) as ei:
            eng._chk(eng._L.pf_adj_segment(eng.h, 0, n, blob.ctypes.data, blob.size, 0))
        assert ei.value.code == N.PF_ERR_NONFINITE
        assert eng.step() == at + 1
        eng._cache.clear()
        assert np.isinf(eng.get("Hx")).any()
    finally:
        eng.close()
