"""Rebuilt contact lists on both sides of the row length up to which a list is
filled as it is counted (32), and past the 256 entries that are sorted in
local memory, in three particle orders: equal to the oracle's at each step."""
import numpy as np
import pytest

from cabanapd_b200 import problems as P

pytestmark = pytest.mark.gpu

CUTOFF = 2 * 1.1e-3 + 0.22e-3


def _points(order, n, mean):
    """About n points with about `mean` others within the cutoff of each."""
    rng = np.random.Generator(np.random.PCG64([n, int(mean)]))
    side = (n * 4.0 / 3.0 * P.PI * CUTOFF ** 3 / mean) ** (1.0 / 3.0)
    if order == "random":
        return rng.uniform(0.0, side, (n, 3))
    k = round(n ** (1.0 / 3.0))
    a = (np.arange(k) + 0.5) * side / k
    x = np.stack(np.meshgrid(a, a, a, indexing="ij"), -1).reshape(-1, 3)  # z fastest
    if order == "x fastest":
        x = x[:, ::-1].copy()
    return x + rng.uniform(-0.02, 0.02, x.shape) * side / k


@pytest.mark.parametrize("order", ["random", "x fastest", "z fastest"])
@pytest.mark.parametrize("n,mean", [(1000, 0.5), (1000, 8), (1728, 28), (1331, 46), (729, 600)])
def test_rebuilt_rows_equal_the_oracles(oracle, order, n, mean):
    import cabanapd_b200
    x = _points(order, n, mean)
    n = len(x)
    params = dict(pd_model=0, contact_model=P.CONTACT_HERTZ, contact_radius=1.1e-3,
                  radius_extend=0.22e-3, nu=0.3, E=7e7, restitution=0.8, dt=1e-5,
                  rebuild_every=1, per_particle_radius=1)
    radius = np.full(n, 1e-5)  # (no overlap: the points move on straight lines)
    # Drawn together, so that rows outgrow the earlier build's.
    centre = x.mean(0)
    prob = dict(params=params, x=x, vol=4.0 / 3.0 * P.PI * radius ** 3, rho=np.full(n, 2500.0),
                nofail=None, radius=radius, u0=None, v0=-400.0 * (x - centre), notches=None,
                bcs=[], n_frozen=0)
    g = P.setup(cabanapd_b200.System(dict(params), precision=1), prob)
    o = P.setup(oracle.OracleSystem(params), prob)
    for _ in range(8):
        g.run(1)
        o.run(1)
        gc, gi, _ = g.neighbors()
        oc, oi, _ = o.neighbors()
        assert np.array_equal(gc, oc)
        m = int(oc.max())
        assert np.array_equal(gi[:, :m], oi[:, :m])
    assert (m > 256) == (mean > 256) and (mean != 46 or m > 32)
