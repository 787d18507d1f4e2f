"""State blobs of grids whose rows are padded, or whose z layers lie in groups.

The blob is compact whatever the layout. Its fields must be the engine's
fields, its z-layer CPML state (after one step from zero state: c times the
quotient, where c is not 0) the one computed here, and it must come out and go
back in the same way through host memory and through device memory at any
byte offset.
"""
import numpy as np
import pytest

import photonfdtd_b200 as pf
from photonfdtd_b200 import _native as N
from photonfdtd_b200.engine import B200Engine, build_tables

pytestmark = pytest.mark.gpu

ALL6 = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")


@pytest.mark.parametrize("precision", ["float32", "float64"])
@pytest.mark.parametrize("shape,pml", [((12, 9, 4), 0), ((11, 13, 5), 0), ((14, 12, 23), 4),
                                       ((16, 17, 32), (4, 4, 5)), ((13, 14, 30), (0, 3, 6)),
                                       ((40, 1, 33), (4, 0, 5)), ((36, 35, 1), (4, 4, 0))])
def test_blob_rows(shape, pml, precision):
    import torch
    d = 20e-9
    pml = (pml,) * 3 if isinstance(pml, int) else pml
    grid = pf.Grid(size=tuple(n * d if n > 1 else 0.0 for n in shape),
                   cell_size=tuple(d if n > 1 else 0.0 for n in shape), pml_layers=pml)
    dt = 0.9 * d / (pf.C_0 * 3 ** 0.5)
    t = build_tables(pf.Simulation(grid, run_time=9.5 * dt, precision=precision))
    rng = np.random.default_rng(8)
    fields = {c: rng.standard_normal(shape).astype(precision) for c in ALL6}
    cells = int(np.prod(shape))
    a, b = B200Engine(t), B200Engine(t)
    try:
        for c in ALL6:
            a.set_field(c, fields[c])
        a.advance(0, 1)
        blob = a.get_state()
        v = blob.view(precision)
        for q, c in enumerate(ALL6):
            np.testing.assert_array_equal(v[q * cells:(q + 1) * cells].reshape(shape), a.get(c))
        # Hx's term along z: E psi first (six arrays), then Hx along y, Hx along z
        per = lambda k, ax: cells // shape[ax] * int(np.count_nonzero(t["cpml"][ax][k]))  # noqa: E731
        axes = (1, 2, 2, 0, 0, 1)
        at = 6 * cells + sum(per(1, ax) for ax in axes) + per(3, 1)
        if shape[1] > 1 and shape[2] > 1:
            ch = np.asarray(t["cpml"][2][3], dtype=precision)
            want = np.zeros(shape, precision)
            ey = fields["Ey"]
            want[:, :-1, :-1] = (ch[:-1] * ((ey[:, :, 1:] - ey[:, :, :-1])
                                            / np.asarray(d, precision)))[:, :-1]
            want = want[:, :, np.flatnonzero(ch)]
            np.testing.assert_array_equal(v[at:at + want.size].reshape(want.shape), want)
        # through device memory, at offsets of every remainder
        for off in (0, 1, 4, 6, 8):
            buf = torch.full((blob.size + 16,), 255, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            a.get_state_to(buf.data_ptr() + off, blob.size)
            got = buf.cpu().numpy()
            np.testing.assert_array_equal(got[off:off + blob.size], blob)
            assert (got[:off] == 255).all() and (got[off + blob.size:] == 255).all()
            for c in ALL6:
                b.set_field(c, np.zeros(shape, precision))
            N.check(N.lib().pf_set_state(b.h, 1, buf.data_ptr() + off, blob.size, 1), b.h)
            b._cache.clear()
            np.testing.assert_array_equal(b.get_state(), blob)
        b.set_state(1, blob)
        np.testing.assert_array_equal(b.get_state(), blob)
        a.advance(1, 5)
        b.advance(1, 5)
        np.testing.assert_array_equal(a.get_state(), b.get_state())
    finally:
        a.close()
        b.close()


def test_fields_larger_than_the_staging_buffer():
    """72 million cells, 289 MB a field: two pieces of the staging buffer."""
    shape = (300, 600, 401)
    d = 20e-9
    grid = pf.Grid(size=tuple(n * d for n in shape), cell_size=d, pml_layers=0)
    t = build_tables(pf.Simulation(grid, run_time=1e-16, precision="float32"))
    f = np.random.default_rng(1).standard_normal(shape, dtype=np.float32)
    eng = B200Engine(t)
    try:
        eng.set_field("Ey", f)
        eng._cache.clear()
        np.testing.assert_array_equal(eng.get("Ey"), f)
        assert not eng.get("Ex").any() and not eng.get("Ez").any()
    finally:
        eng.close()
