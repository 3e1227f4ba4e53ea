"""The exact kernels' shared-iteration roots and quotients give the IEEE
results: forces, energies and LPS fields bit for bit the oracle's on clouds
whose lengths and force factors lie in the middle of the exponent range, at
its ends and beyond (where the IEEE operations take over), with coincident
displacements (zero components) and undeformed bonds."""
import numpy as np
import pytest

from cabanapd_b200 import problems as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda():
    import cabanapd_b200
    return cabanapd_b200


def _cloud(model, fracture, scale, factor, n, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    x = rng.uniform(0.0, 1.0, (n, 3))
    u0 = rng.normal(0.0, 0.02, (n, 3))
    u0[rng.random(n) < 0.3] = 0.0   # undeformed bonds, zero components
    u0[:, 2] *= rng.random(n) < 0.5
    params = dict(pd_model=model, fracture=int(fracture), horizon=0.35 * scale, K=factor, G=0.5 * factor,
                  G0=factor * scale * 1e-2, dt=1.0)
    return dict(params=params, x=x * scale, vol=rng.uniform(0.5, 2.0, n) / n, rho=None, nofail=None,
                radius=None, u0=u0 * scale, v0=None, notches=None, bcs=[], n_frozen=0)


@pytest.mark.parametrize("model,fracture", [(P.PD_PMB, False), (P.PD_PMB, True), (P.PD_LPS, False),
                                            (P.PD_LPS, True)])
@pytest.mark.parametrize("scale,factor", [(1.0, 1.0), (1e-3, 1e11), (1e60, 1.0), (1e-70, 1e-30),
                                          (1.0, 1e-160), (1.0, 1e200)])
def test_exact_results_over_the_exponent_range(cuda, oracle, model, fracture, scale, factor):
    prob = _cloud(model, fracture, scale, factor, 700, 5)
    g = cuda.System(dict(prob["params"]))
    c = oracle.OracleSystem(prob["params"])
    for s in (g, c):
        P.setup(s, prob)
        s.compute_energy()
    names = ["f", "W"] + (["m", "theta"] if model == P.PD_LPS else [])
    for name in names + (["phi"] if fracture else []):
        a, b = g.get(name), c.get(name)
        assert np.array_equal(a, b, equal_nan=True), name
    if fracture:
        assert np.array_equal(g.neighbors()[2], c.neighbors()[2])
