"""The lattice walks on both sides of the sizes where their block changes
(148 SMs; 256 threads up to 148 x 256 rows, 512 from there, 256 again past
148 x 512, 512 past 148 x 768): fields and bonds against the oracle, with the
bars of the precisions, and one row less and more than the whole blocks."""
import numpy as np
import pytest

from cabanapd_b200 import problems as P

pytestmark = pytest.mark.gpu


def _nrel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.fixture(scope="module")
def solved(oracle):
    """The oracle after ten steps of a body of cells, each body once."""
    done = {}

    def solve(cells):
        if cells not in done:
            nx, ny, nz = cells
            prob = P.plate_impact(num_cells=cells, steps=10, v0=60.0,
                                  size=(0.2, 0.2 * ny / nx, 0.2 * nz / nx))
            o = P.setup(oracle.OracleSystem(prob["params"]), prob)
            o.run(10)
            done[cells] = (prob, {f: o.get(f) for f in ("u", "v", "f")}, o.neighbors()[2])
        return done[cells]

    return solve


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("cells", [(33, 31, 37), (64, 37, 16), (71, 67, 8), (148, 64, 8),
                                   (149, 64, 8), (96, 74, 16), (97, 74, 16)])
def test_bodies_at_the_block_sizes_edges(solved, cells, precision):
    import cabanapd_b200
    prob, want, bonds = solved(cells)
    g = P.setup(cabanapd_b200.System(dict(prob["params"], precision=precision)), prob)
    warps, irregular, _ = g.stencil_stats()
    assert warps == (cells[0] * cells[1] * cells[2] + 31) // 32 and irregular == 0
    g.run(10)
    assert np.array_equal(g.neighbors()[2], bonds)
    bars = dict(u=1e-12, v=1e-12, f=1e-12) if precision == 1 else dict(u=1e-6, v=1e-5, f=1e-5)
    for name, bar in bars.items():
        assert _nrel(g.get(name), want[name]) <= bar, name
