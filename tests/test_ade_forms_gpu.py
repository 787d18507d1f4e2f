"""The two forms of the dispersive E pass against the oracle, bit for bit.

The vector form suits scenes whose polarisation records form aligned runs, the
one-cell form all others; the engine decides by counting warps. Blocks at
aligned positions take the first, scattered cells and blocks on rows that
break the alignment the second (pf_info tells), for media of one, two and three
poles, with layers and without, at row lengths of every remainder.
"""
import numpy as np
import pytest

import photonfdtd_b200 as pf
from photonfdtd_b200.engine import B200Engine, build_tables
from test_split3d_gpu import ALL6, _box

pytestmark = pytest.mark.gpu


def _scene(shape, precision, block, pml, d, n_media):
    rng = np.random.default_rng(5)
    grid = pf.Grid(size=tuple(n * d for n in shape), cell_size=d, pml_layers=pml)
    dt = 0.99 * d / (pf.C_0 * 3 ** 0.5)
    u = 0.2 / dt
    pole = [pf.Pole(strength=(u * s) ** 2, omega0=u * w, gamma=u * 0.01)
            for s, w in ((1.0, 0.0), (0.5, 0.4), (0.3, 0.7))]
    mats = [pf.DispersiveMedium(eps_inf=1.0 + q, poles=tuple(pole[:q + 1])) for q in range(3)]
    structures = []
    for lo in np.ndindex(*[-(-n // block) for n in shape]):
        m = int(rng.integers(0, n_media + 1 if block > 1 else 9))
        if m < n_media:
            lo = [block * v for v in lo]
            hi = [min(v + block, n) for v, n in zip(lo, shape)]
            structures.append(_box(shape, d, lo, hi, mats[m]))
    return pf.Simulation(grid, structures=structures, run_time=9.5 * dt, precision=precision)


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("shape,block,pml,d,n_media,form", [
    ((64, 16, 64), 16, 0, 20e-9, 3, "cell"), ((33, 14, 31), 5, 4, 20e-9, 3, "cell"),
    ((12, 13, 14), 1, (3, 0, 4), 13e-9, 3, "cell"), ((17, 16, 33), 3, 4, 200e-9, 3, "cell"),
    ((48, 24, 48), 8, 6, 20e-9, 1, "vector"), ((20, 24, 43), 24, 5, 20e-9, 1, "vector")])
def test_both_forms_bitwise_against_oracle(shape, block, pml, d, n_media, form, precision):
    from oracle import OracleRun
    sim = _scene(shape, precision, block, pml, d, n_media)
    rng = np.random.default_rng(7)
    lo = -40.0 if precision == "float32" else -290.0
    fields = {c: (rng.standard_normal(shape) * 10.0 ** rng.uniform(lo, 3.0, size=shape))
              .astype(precision) for c in ALL6}
    eng = B200Engine(build_tables(sim))
    try:
        assert eng.info()["e_pass"] == form
        eng.set_profiling(True)  # separate passes
        for c in ALL6:
            eng.set_field(c, fields[c])
        eng.advance(0, 4)
        assert eng.read_profile()[0][0] == 8
        got = {c: eng.get(c).copy() for c in ALL6}
    finally:
        eng.close()
    run = OracleRun(sim)
    run.set_fields(fields)
    run.advance(4)
    for c in ALL6:
        np.testing.assert_array_equal(got[c], run.F[c], err_msg=c)
