"""The stencil warp lists of a body that is one box of lattice lines: every
warp once, whatever the box's sides leave over of the tiles, and nothing but
the body decides their order."""
import os
import subprocess
import sys

import numpy as np
import pytest

from cabanapd_b200 import problems as P

pytestmark = pytest.mark.gpu

STEPS = 4

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _plate(cells, frozen=0):
    nx, ny, nz = cells
    prob = P.plate_impact(num_cells=cells, steps=STEPS, v0=60.0,
                          size=(0.2, 0.2 * ny / nx, 0.2 * nz / nx))
    prob["n_frozen"] = frozen
    return prob


# (Planes of 240 thousand rows on are walked in tiles of 4 x 4 lines.)
@pytest.mark.parametrize("cells,frozen", [((97, 13, 7), 97 * 3 + 40), ((600, 399, 2), 0),
                                          ((600, 400, 2), 0), ((613, 397, 5), 0),
                                          ((613, 393, 3), 613 * 3 + 40)])
def test_every_row_is_advanced(oracle, cells, frozen):
    """A warp left out or taken twice leaves whole rows off by their own size;
    the FP64 path's bar is 1e-12 norm-wise."""
    import cabanapd_b200
    prob = _plate(cells, frozen)
    g = cabanapd_b200.System(dict(prob["params"], precision=1))
    o = oracle.OracleSystem(prob["params"])
    for s in (g, o):
        P.setup(s, prob)
    warps, irregular, _ = g.stencil_stats()
    assert warps + irregular == (len(prob["x"]) - frozen + 31) // 32
    g.run(STEPS)
    o.run(STEPS)
    for name in ("u", "v", "f"):
        a, b = g.get(name), o.get(name)
        assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b), name


PROGRAM = """
import sys
sys.path.insert(0, sys.argv[1])
import cabanapd_b200
from cabanapd_b200 import problems as P
prob = P.plate_impact(num_cells=(600, 405, 4), steps=3, v0=60.0, size=(0.2, 0.135, 0.2 * 4 / 600))
s = cabanapd_b200.System(dict(prob["params"], precision=2))
P.setup(s, prob)
print(" ".join(v.hex() for v in s.step_energy(3)))
"""


@pytest.mark.parametrize("value", ["1", "x"])
def test_totals_do_not_depend_on_the_callers_environment(value):
    """The order of the warps is the order of the energy partials, so the
    totals' last bits show it."""
    def totals(env):
        return subprocess.run([sys.executable, "-c", PROGRAM, ROOT], env=dict(os.environ, **env),
                              check=True, capture_output=True, text=True, timeout=300).stdout
    assert totals({}) == totals({"T_Y": value, "T_Z": value})
