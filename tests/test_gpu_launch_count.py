"""cpd_kernel_launches of a step on the lattice-stencil kernels, exactly."""
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

