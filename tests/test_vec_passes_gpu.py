"""The 3D vector passes against the oracle, bit for bit.

The scenes of test_split3d_gpu.py are small enough for resident launches,
which the engine takes by itself. Profiling (pf_set_profiling) makes it launch
every pass alone; the launch counters show that it did (two step passes per
step), and that by default it does not.
"""
import numpy as np
import pytest

from photonfdtd_b200.engine import B200Engine, build_tables
from test_split3d_gpu import ALL6, _scene

import photonfdtd_b200 as pf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("media", ["cell", "tensor", "blocks", "scattered"])
@pytest.mark.parametrize("shape,pml,d", [((40, 37, 64), 6, 20e-9), ((21, 70, 101), 5, 13e-9),
                                         ((18, 23, 35), (4, 0, 6), 47e-9),
                                         ((30, 9, 130), (0, 0, 0), 20e-9),
                                         ((24, 20, 39), 5, 200e-9)])
def test_separate_passes_bitwise_against_oracle(shape, pml, d, media, precision):
    from oracle import OracleRun
    sim = _scene(shape, precision, media, pml, d)
    rng = np.random.default_rng(7)
    ce3 = None
    if media == "tensor":
        base = sim.dt / pf.EPS_0
        ce3 = [(base * rng.uniform(0.1, 1.0, size=shape)).astype(precision) for _ in range(3)]
    lo = -40.0 if precision == "float32" else -310.0
    fields = {}
    for c in ALL6:
        mag = 10.0 ** rng.uniform(lo, 3.0, size=shape)
        fields[c] = (rng.standard_normal(shape) * mag).astype(precision)
    run = OracleRun(sim, ce3=ce3)
    run.set_fields(fields)
    run.advance(3)
    t = build_tables(sim, ce3=ce3)
    for separate in (True, False):
        eng = B200Engine(t)
        try:
            eng.set_profiling(separate)
            for c in ALL6:
                eng.set_field(c, fields[c])
            eng.advance(0, 3)
            assert eng.read_profile()[0][0] == (6 if separate else 1)
            for c in ALL6:
                np.testing.assert_array_equal(eng.get(c), run.F[c], err_msg=f"{c} {separate}")
        finally:
            eng.close()
