"""Memory kept from destroyed engines goes back when it is wanted.

The memory of a destroyed engine stays mapped for the next one (up to 2 GiB).
A batch that sizes its checkpoints by the free memory must see it as free, and
pf_release_memory gives it back to other users of the device.
"""
import pytest

import photonfdtd_b200 as pf
from photonfdtd_b200 import _native as N
from photonfdtd_b200.batch import default_memory_budget
from photonfdtd_b200.engine import B200Engine, build_tables

pytestmark = pytest.mark.gpu

SLACK = 64 << 20  # what the context itself may take meanwhile


def _engine_come_and_gone():
    d, n = 20e-9, 256
    grid = pf.Grid(size=(n * d,) * 3, cell_size=d, pml_layers=8)
    t = build_tables(pf.Simulation(grid, run_time=1e-15, precision="float32"))
    eng = B200Engine(t)
    try:
        eng.advance(0, 2)
        return eng.device_bytes()
    finally:
        eng.close()


def test_a_batch_sees_the_kept_memory_as_free():
    import torch
    _engine_come_and_gone()
    before = 2.0 * default_memory_budget()
    held = _engine_come_and_gone()
    assert 4 * SLACK < held < 2 << 30
    assert torch.cuda.mem_get_info()[0] <= before - held + SLACK  # kept
    assert 2.0 * default_memory_budget() >= before - SLACK


def test_release_memory():
    import torch
    held = _engine_come_and_gone()
    kept = torch.cuda.mem_get_info()[0]
    N.check(N.lib().pf_release_memory())
    assert torch.cuda.mem_get_info()[0] >= kept + held - SLACK
    N.check(N.lib().pf_release_memory())  # nothing left: no error
    _engine_come_and_gone()
