"""The exact kernels where their shared iterations give way to the IEEE
operations: squared lengths past both ends of the range, roots next to a
midpoint of two doubles, lengths whose low word is all ones, a length of zero.
Fields and bonds bit for bit the oracle's."""
import math
import struct
from fractions import Fraction

import numpy as np
import pytest

from cabanapd_b200 import problems as P

pytestmark = pytest.mark.gpu

MODELS = [(P.PD_PMB, False), (P.PD_PMB, True), (P.PD_LPS, False), (P.PD_LPS, True)]


def _next_to_midpoints(count):
    """Doubles in [1, 4) whose root is within 2^-25 of a unit of a midpoint: with
    the midpoint (m + 1/2) 2^-52, m (m + 1) a little over a multiple of 2^53."""
    out = []
    for c in range(2, 2 + 2 * count, 2):
        m = 1  # m (m + 1) = c mod 2^k, lifted bit by bit
        if (m * (m + 1) - c) % 4:
            m = 0
        for k in range(2, 54):
            if (m * (m + 1) - c) % (1 << (k + 1)):
                m += 1 << k
        m = (m & ((1 << 53) - 1)) | (1 << 52)
        square = m * (m + 1) - c
        shift = square.bit_length() - 53
        if square % (1 << shift):
            continue
        a = float(Fraction(square, 1 << 104))
        root = Fraction(math.isqrt(int(Fraction(a) * (1 << 160))), 1 << 80)
        assert abs(root - Fraction(2 * m + 1, 1 << 53)) * (1 << 52) < Fraction(1, 1 << 25)
        out.append(a)
    assert len(out) > count // 4
    return out


def _vector(a):
    """x, y with x x + y y == a as rounded (y about half as long)."""
    for step in range(1, 4000):
        x = math.sqrt(a) * (0.8 + step * 1e-5)
        y = math.sqrt(a - x * x)
        for _ in range(8):
            if x * x + y * y == a:
                return (x, y, 0.0)
            y = math.nextafter(y, math.inf if x * x + y * y < a else 0.0)
    raise AssertionError(a)


def _vectors(kind):
    if kind == "midpoint":
        below = [math.nextafter(4.0 ** k, 0.0) for k in (-1, 0, 1)]
        assert all(math.sqrt(a) < 2.0 ** k for a, k in zip(below, (-1, 0, 1)))
        return [_vector(a) for a in below + _next_to_midpoints(64)]
    # One-axis lengths whose low word is all ones.
    rng = np.random.Generator(np.random.PCG64(3))
    out = []
    for k in range(48):
        high = struct.pack("<I", 0x3ff00000 + int(rng.integers(0x100000)))
        v = [0.0, 0.0, 0.0]
        v[k % 3] = struct.unpack("<d", b"\xff\xff\xff\xff" + high)[0] * (-1) ** k
        out.append(tuple(v))
    return out


def _compare(oracle, prob, model, fracture):
    import cabanapd_b200
    g = P.setup(cabanapd_b200.System(dict(prob["params"])), prob)
    o = P.setup(oracle.OracleSystem(prob["params"]), prob)
    for s in (g, o):
        s.compute_energy()
    assert np.array_equal(g.neighbors()[0], o.neighbors()[0]) and o.neighbors()[0].max() > 0
    names = ["f", "W"] + (["m", "theta"] if model == P.PD_LPS else [])
    for name in names + (["phi"] if fracture else []):
        assert np.array_equal(g.get(name), o.get(name), equal_nan=True), name
    if fracture:
        assert np.array_equal(g.neighbors()[2], o.neighbors()[2])
    return o


def _problem(model, fracture, x, u0, horizon, vol, stretch=0.05, influence=1):
    # G0 from the critical stretch s0 = sqrt(5 G0 / (9 K horizon)), K = 1.
    params = dict(pd_model=model, fracture=int(fracture), influence_type=influence,
                  horizon=horizon, K=1.0, G=0.5, G0=1.8 * horizon * stretch ** 2, dt=1.0)
    return dict(params=params, x=x, vol=vol, rho=None, nofail=None, radius=None, u0=u0, v0=None,
                notches=None, bcs=[], n_frozen=0)


@pytest.mark.parametrize("model,fracture", MODELS)
@pytest.mark.parametrize("kind", ["midpoint", "all ones"])
@pytest.mark.parametrize("share", [0.0, 0.5])
def test_constructed_lengths(oracle, model, fracture, kind, share):
    """Particle 0 at the origin; bond (0, k) has vector k as its deformed
    vector, and as its reference one with share 0 (else half of it)."""
    v = np.array([(0.0, 0.0, 0.0)] + _vectors(kind))
    vol = np.linspace(0.5, 1.5, len(v))
    prob = _problem(model, fracture, v * (1.0 - share), v * share, 9.0, vol)
    _compare(oracle, prob, model, fracture)


@pytest.mark.parametrize("model,fracture", MODELS)
@pytest.mark.parametrize("influence", [0, 1])
@pytest.mark.parametrize("scale", [1e140, 1e-140])
def test_lengths_past_the_range(oracle, model, fracture, influence, scale):
    """Squares of 1e280 and 1e-280, the range's ends being 2^900 and 2^-900. (The
    bond constants leave the doubles before that; LPS volumes and dilatations
    and the breaking of bonds do not use them.)"""
    rng = np.random.Generator(np.random.PCG64(11))
    x = rng.uniform(0.0, 1.0, (300, 3))
    u0 = rng.normal(0.0, 0.02, (300, 3))
    prob = _problem(model, fracture, x * scale, u0 * scale, 0.4 * scale,
                    rng.uniform(0.5, 2.0, 300), influence=influence)
    o = _compare(oracle, prob, model, fracture)
    if model == P.PD_LPS:
        assert np.isfinite(o.get("m")).all() and o.get("m").max() > 0.0


@pytest.mark.parametrize("model,fracture", MODELS)
def test_a_deformed_length_of_zero(oracle, model, fracture):
    """A pair pushed onto one point (s = -1, and a force of 0 / 0) among others."""
    rng = np.random.Generator(np.random.PCG64(12))
    x = np.round(rng.uniform(0.0, 1.0, (60, 3)) * 1024) / 1024
    x[3] = 0.5
    x[7] = x[3] + np.array([0.25, -0.125, 0.0])  # (a bond, within the horizon)
    u0 = np.zeros_like(x)
    u0[7] = x[3] - x[7]
    prob = _problem(model, fracture, x, u0, 0.6, np.full(60, 0.01))
    o = _compare(oracle, prob, model, fracture)
    assert np.isnan(o.get("f")).any()
