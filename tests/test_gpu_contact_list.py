"""Contact lists and Hertz forces of random clouds against the oracle: lists
rebuilt every step (filled as they are counted, and refilled when a row
outgrows the list an earlier build left), empty and one-particle rows, sizes
off the warp, both particle orders, equal and per-particle radii."""
import numpy as np
import pytest

from cabanapd_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda():
    import cabanapd_b200
    return cabanapd_b200


def _cloud(n, spread, per_particle, speed, seed):
    """n spheres of about 1 mm at random points of a box of `spread` mm per
    sphere and axis; speed < 0 draws the cloud together."""
    rng = np.random.Generator(np.random.PCG64(seed))
    side = spread * 1e-3 * max(n, 2) ** (1.0 / 3.0)
    x = rng.uniform(-0.5 * side, 0.5 * side, (n, 3))
    radius = rng.uniform(0.9e-3, 1.1e-3, n)
    params = dict(pd_model=0, contact_model=P.CONTACT_HERTZ, contact_radius=1.1e-3,
                  radius_extend=0.22e-3, nu=0.3, E=7e7, restitution=0.8, dt=1e-5,
                  rebuild_every=1, per_particle_radius=int(per_particle))
    return dict(params=params, x=x, vol=4.0 / 3.0 * P.PI * radius ** 3,
                rho=rng.uniform(2000.0, 3000.0, n), nofail=None, radius=radius, u0=None,
                v0=speed * x + rng.normal(0.0, 0.05, (n, 3)), notches=None, bcs=[], n_frozen=0)


def _pair(cuda, oracle, prob, ordering=0):
    g = cuda.System(dict(prob["params"]), precision=1, ordering=ordering)
    c = oracle.OracleSystem(prob["params"])
    return P.setup(g, prob), P.setup(c, prob)


@pytest.mark.parametrize("n,spread,speed,ordering",
                         [(1, 2.0, 0.0, 0), (2, 1.0, 0.0, 0), (33, 6.0, -3000.0, 0),
                          (700, 4.0, -3000.0, 0), (700, 4.0, -3000.0, 1), (1500, 1.1, 0.0, 0)])
def test_rebuilt_lists_equal_the_oracles(cuda, oracle, n, spread, speed, ordering):
    prob = _cloud(n, spread, True, speed, 7 + n)
    g, c = _pair(cuda, oracle, prob, ordering)
    longest = []
    for _ in range(12):
        g.run(1)
        c.run(1)
        gc, gi, _ = g.neighbors()
        cc, ci, _ = c.neighbors()
        assert np.array_equal(gc, cc)
        m = int(cc.max())
        longest.append(m)
        assert np.array_equal(gi[:, :m], ci[:, :m])
    if speed < 0 and n > 100:
        assert longest[-1] > longest[0]  # the list had to grow


@pytest.mark.parametrize("per_particle", [False, True])
@pytest.mark.parametrize("n,spread", [(2, 1.0), (257, 1.2), (1000, 1.7)])
def test_hertz_force_against_the_oracle(cuda, oracle, n, spread, per_particle):
    """Every operation behind the overlap is a rounding or two of a smooth
    law: norm-wise within the contact bar of 1e-12 of the oracle."""
    prob = _cloud(n, spread, per_particle, 0.0, 31 + n)
    if n == 2:  # one overlapping pair
        prob["x"][1] = prob["x"][0] + np.array([1.0e-3, 1.1e-3, -0.7e-3])
    g, c = _pair(cuda, oracle, prob)
    for s in (g, c):
        s.compute_force()
    a, b = g.get("f"), c.get("f")
    assert np.linalg.norm(b) > 0.0
    assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b)
