"""cpd_kernel_launches of a step on the lattice-stencil kernels, exactly, and
the device bytes that the FP64 tables hold."""
import ctypes

import pytest

from cabanapd_b200 import problems as P

pytestmark = pytest.mark.gpu

CELLS = (96, 48, 8)


def _system(precision, horizon_factor=3.01):
    import cabanapd_b200
    prob = P.plate_impact(num_cells=CELLS, steps=20, v0=60.0, size=(0.2, 0.1, 0.2 * 8 / 96),
                          horizon_factor=horizon_factor)
    return P.setup(cabanapd_b200.System(dict(prob["params"], precision=precision)), prob)


# First half step; FP64: the gather records; then the walk's launches per step
# (one, or one per 64 entries of a wide table).
@pytest.mark.parametrize("precision,horizon_factor,entries,before,per_step",
                         [(1, 3.01, 122, 2, 1), (2, 3.01, 122, 1, 1), (1, 4.0, 256, 2, 4)])
def test_launches_of_a_step(precision, horizon_factor, entries, before, per_step):
    s = _system(precision, horizon_factor)
    warps, irregular, found = s.stencil_stats()
    assert (warps > 0, irregular, found) == (True, 0, entries)
    s.step(1)
    for steps in (1, 7):
        counted = s.kernel_launches()
        s.step(steps)
        assert s.kernel_launches() - counted == before + per_step * steps


def _bytes(system):
    system.step(1)
    n = ctypes.c_uint64()
    assert system._lib.cpd_device_bytes(system._h, ctypes.byref(n)) == 0
    return n.value


@pytest.mark.parametrize("horizon_factor,layers,parts", [(3.01, 3, 0), (4.0, 4, 1)])
def test_partial_forces_are_held_for_wide_tables_only(horizon_factor, layers, parts):
    """Beyond the exact path's: the second displacement (24 bytes a row), two
    buffers of 32-byte records with guards of the farthest offset, presence
    masks of 4 bytes per 32 entries, lists and masks per warp (under 4 bytes a
    row), and 32 bytes a row of partial forces where the walk has parts."""
    rows = CELLS[0] * CELLS[1] * CELLS[2]
    records = rows + 2 * (layers * CELLS[0] * CELLS[1] + 32)
    masks = 16 if horizon_factor < 4 else 32
    least = (24 + masks + 32 * parts) * rows + 64 * records
    held = _bytes(_system(1, horizon_factor)) - _bytes(_system(0, horizon_factor))
    assert least <= held <= least + 8 * rows
