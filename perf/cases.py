"""Performance cases: time steps, output steps, batches and whole jobs.

Every case is one body of particles taken a number of time steps through the
public Python binding (System, Batch, problems.setup). Kinds:

  wave      elastic PMB cube with a radial displacement pulse (the elastic
            wave program, 41^3 in the benchmark)
  plate     PMB fracture, double-notched plate under impact, mid-run: the
            body carries strain waves of a fair part of the critical stretch.
            `horizon` is delta / dx (3.01; the example decks also use 4).
            `layout` "deck" takes the plate's own 0.2 x 0.1 x 0.009 m for any
            cell counts (unequal spacings), "cubic" equal spacings
  box       LPS fracture, random pre-notches, traction on the y faces
  packing   Hertzian spheres, list rebuilt every 10 steps: "settled" (simple
            cubic, every contact slightly compressed) or "dilute" (jittered,
            spheres apart)
  cylinder  PMB fracture with normal-repulsion contact, particles at random
            points of their cells (the fragmenting cylinder)
  batch     small wave / plate / box bodies advanced together
  job       a whole plate job from host arrays: set-up, steps with an output
            step every 10, displacements back to the host, closing

`steps` is the number of time steps of one pass; with `output` the pass ends
in an output step (energy and damage totals).

exact() integrates the same equations in plain float64 torch: bodies sit on a
grid of cells, so each bond or contact is a grid offset and every sum is a
loop over offsets of shifted arrays.
"""
import math

import numpy as np
import torch

import cabanapd_b200
from cabanapd_b200 import problems

PRECISION = {"exact": 0, "fp64": 1, "mixed": 2}
PMB, LPS = 1, 2


# ---------------------------------------------------------------------------
# The cases.

def listed():
    return [
        # The smallest bodies: launches and latency count.
        dict(name="wave_4k_fp64", kind="wave", nx=16, ny=16, nz=16, precision="fp64", steps=20,
             output=False),
        # The elastic-wave benchmark's body (41^3).
        dict(name="wave_69k_mixed", kind="wave", nx=41, ny=41, nz=41, precision="mixed",
             steps=20, output=False),
        # The Kalthoff-Winkler deck's size in the binding's default precision.
        dict(name="plate_79k_exact", kind="plate", layout="deck", nx=151, ny=75, nz=7,
             horizon=3.01, precision="exact", steps=10, output=True),
        # The 1.2 M-particle plate, plain FP64, an output step every 10.
        dict(name="plate_1m2_fp64", kind="plate", layout="deck", nx=376, ny=188, nz=17,
             horizon=3.01, precision="fp64", steps=10, output=True),
        # The benchmark's full plate, mixed precision, an output step every 10.
        dict(name="plate_11m5_mixed", kind="plate", layout="deck", nx=800, ny=400, nz=36,
             horizon=3.01, precision="mixed", steps=10, output=True),
        # The crack-branching lattice at the example decks' four-spacing horizon.
        dict(name="plate_512k_h4_fp64", kind="plate", layout="cubic", nx=400, ny=160, nz=8,
             horizon=4.01, precision="fp64", steps=10, output=False),
        # LPS fracture, plain FP64, mid size.
        dict(name="box_1m_fp64", kind="box", nx=500, ny=200, nz=10, precision="fp64", steps=10,
             output=False),
        # The LPS benchmark's box, mixed precision.
        dict(name="box_8m_mixed", kind="box", nx=1000, ny=400, nz=20, precision="mixed", steps=4,
             output=False),
        # The DEM benchmark's size, every sphere in contact with its neighbours.
        dict(name="packing_4m_fp64", kind="packing", layout="settled", nx=200, ny=200, nz=100,
             precision="fp64", steps=20, output=False),
        # The fragmenting cylinder's deck: off-lattice bonds and contact.
        dict(name="cylinder_fp64", kind="cylinder", across=50, precision="fp64", steps=5,
             output=False),
        # Many small specimens advanced together (as the job server batches them).
        dict(name="batch_16_mixed", kind="batch", jobs=16, largest=20000, precision="mixed",
             steps=16, output=False),
        # A whole mid-size job: set-up, 100 steps with outputs, results back.
        dict(name="job_1m4_mixed", kind="job", layout="cubic", nx=400, ny=200, nz=18,
             horizon=3.01, precision="mixed", steps=100, output=True),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["wave", "plate", "plate", "box", "packing", "cylinder", "batch", "job"])
    pick = rng.choice(["fp64", "fp64", "mixed", "mixed", "exact"])
    case = dict(kind=kind, precision=pick, steps=rng.randint(5, 24), output=rng.random() < 0.3)
    if kind == "wave":
        s = _log(rng, 4e3, 1.5e6) ** (1 / 3)
        case.update(nx=round(s), ny=max(8, round(s * rng.uniform(0.8, 1.2))), nz=round(s))
    elif kind in ("plate", "job"):
        n = _log(rng, 2e4, 2e6)
        case.update(layout=rng.choice(["deck", "cubic"]), horizon=rng.choice([3.01, 3.01, 4.01]))
        a = (n / (0.5 * 0.045)) ** (1 / 3)
        case.update(nx=round(a), ny=round(a / 2 * rng.uniform(0.9, 1.1)),
                    nz=max(3, round(0.045 * a)))
        if kind == "job":
            case.update(precision=rng.choice(["fp64", "mixed"]), steps=10 * rng.randint(2, 10),
                        output=True)
    elif kind == "box":
        a = (_log(rng, 2e4, 3e6) / (0.4 * 0.02)) ** (1 / 3)
        case.update(nx=round(a), ny=round(0.4 * a), nz=max(3, round(0.02 * a)))
    elif kind == "packing":
        s = _log(rng, 2e4, 4e6) ** (1 / 3)
        case.update(layout=rng.choice(["settled", "dilute"]), nx=round(s),
                    ny=max(8, round(s * rng.uniform(0.8, 1.2))), nz=round(s), output=False)
    elif kind == "cylinder":
        case.update(across=rng.randint(36, 64), steps=rng.randint(2, 6), output=False)
    else:
        case.update(jobs=rng.randint(4, 20), largest=round(_log(rng, 5e3, 3e4)),
                    precision=rng.choice(["fp64", "mixed"]), output=False)
    return case


# ---------------------------------------------------------------------------
# Bodies: a problem dict for problems.setup, on a grid of cells (x fastest).

def _grid(nx, ny, nz, size):
    """Cell-centre coordinates per axis (centred box), spacings."""
    axes, h = [], []
    for n, s in zip((nx, ny, nz), size):
        low, d = -0.5 * s, s / n
        i = np.arange(n, dtype=np.float64)
        lo = low + i * d
        axes.append(lo + 0.5 * ((low + (i + 1.0) * d) - lo))
        h.append(d)
    return axes, h


def _points(axes):
    n = [len(a) for a in axes]
    x = np.empty((n[2], n[1], n[0], 3))
    x[..., 0] = axes[0][None, None, :]
    x[..., 1] = axes[1][None, :, None]
    x[..., 2] = axes[2][:, None, None]
    return x.reshape(-1, 3)


def _waves(rng, axes, size, peak):
    """A smooth random vector field whose gradient is at most about `peak`."""
    n = [len(a) for a in axes]
    out = np.zeros((n[2], n[1], n[0], 3))
    for c in range(3):
        for _ in range(2):
            k = [rng.uniform(1.0, 4.0) * math.pi / size[0] for _ in range(3)]
            s = [np.sin(k[d] * axes[d] + rng.uniform(0, 2 * math.pi)) for d in range(3)]
            a = peak / 6.0 / max(k)
            out[..., c] += a * s[0][None, None, :] * s[1][None, :, None] * s[2][:, None, None]
    return out.reshape(-1, 3)


def _body(case, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    return {"wave": _wave, "plate": _plate, "job": _plate, "box": _box, "packing": _packing,
            "cylinder": _cylinder}[case["kind"]](case, rng)


def _problem(params, x, grid, h, vol, rho, **kw):
    n = x.shape[0]
    full = lambda v: np.full(n, float(v)) if np.isscalar(v) else v  # noqa: E731
    p = dict(params=params, x=x, vol=full(vol), rho=full(rho), nofail=None, radius=None, u0=None,
             v0=None, notches=None, bcs=[], n_frozen=0, grid=grid, h=h, cell=None, bc=None)
    p.update(kw)
    return p


def _wave(case, rng):
    grid = (case["nx"], case["ny"], case["nz"])
    axes, h = _grid(*grid, [1.0 * n / grid[0] for n in grid])
    x = _points(axes)
    centre = rng.uniform(-0.1, 0.1, 3)
    d = x - centre
    r = np.sqrt((d * d).sum(1))[:, None]
    u0 = rng.uniform(0.5, 1.5) * 1e-4 * np.exp(-(r / 0.1) ** 2) * d / np.maximum(r, 1e-30)
    params = dict(pd_model=PMB, fracture=0, horizon=3.01 * h[0], K=1.0, dt=0.3 * h[0])
    return _problem(params, x, grid, h, h[0] * h[1] * h[2], 1.0, u0=u0,
                    v0=_waves(rng, axes, [1.0], 1e-4))


def _plate(case, rng):
    grid = (case["nx"], case["ny"], case["nz"])
    if case["layout"] == "deck":
        size = [0.2, 0.1, 0.009]
    else:
        size = [0.2 * n / grid[0] for n in grid]
    axes, h = _grid(*grid, size)
    x = _points(axes)
    E, nu, rho, G0 = 191e9, 0.25, 8000.0, 22170.0
    K = E / (3.0 * (1.0 - 2.0 * nu))
    horizon = case["horizon"] * h[0]
    s0 = math.sqrt(5.0 * G0 / 9.0 / K / horizon)
    low = [-0.5 * s for s in size]
    y1, y2 = -size[1] / 4.0, size[1] / 4.0
    p0 = np.array([[low[0], y1, low[2]], [low[0], y2, low[2]]])
    v1 = np.array([[size[0] / 4.0, 0.0, 0.0]] * 2)
    v2 = np.array([[0.0, 0.0, size[2]]] * 2)
    strip = np.nonzero((x[:, 0] < low[0] + h[0]) & (x[:, 1] > y1) & (x[:, 1] < y2))[0]
    v0 = _waves(rng, axes, size, 0.6 * s0 * 5000.0)
    v0[strip, 0] = rng.uniform(12.0, 20.0)
    params = dict(pd_model=PMB, fracture=1, horizon=horizon, K=K, G0=G0, dt=0.25 * h[0] / 5000.0)
    return _problem(params, x, grid, h, h[0] * h[1] * h[2], rho,
                    u0=_waves(rng, axes, size, 0.6 * s0), v0=v0, notches=(v1, v2, p0),
                    bcs=[(0, 0, strip, np.array([0.0]))], bc=("zero", strip, None))


def _box(case, rng):
    grid = (case["nx"], case["ny"], case["nz"])
    size = [0.1, 0.04, 0.002]
    axes, h = _grid(*grid, size)
    x = _points(axes)
    horizon = 3.01 * h[0]
    K, G, rho, G0 = 14.9e9, 8.9e9, 2440.0, 3.8
    s0 = math.sqrt(8.0 * G0 / 15.0 / K / horizon)
    k = 20
    p0 = np.stack([rng.uniform(-0.04, 0.04, k), rng.uniform(-0.01, 0.01, k),
                   np.full(k, -0.5 * size[2])], 1)
    length, angle = rng.uniform(0.002, 0.01, k), rng.uniform(0.0, math.pi, k)
    v1 = np.stack([length * np.cos(angle), length * np.sin(angle), np.zeros(k)], 1)
    v2 = np.stack([np.zeros(k), rng.uniform(-1.0, 1.0, k) * size[2], np.full(k, size[2])], 1)
    y = x[:, 1]
    nofail = (np.abs(y) >= 0.5 * size[1] - horizon).astype(np.int32)
    pulled = np.nonzero(np.abs(y) >= 0.5 * size[1] - h[1])[0]
    load = 2e6 / h[1] * np.sign(y[pulled])
    params = dict(pd_model=LPS, fracture=1, influence_type=0, horizon=horizon, K=K, G=G, G0=G0,
                  dt=0.2 * h[0] / 3500.0)
    return _problem(params, x, grid, h, h[0] * h[1] * h[2], rho, nofail=nofail,
                    u0=_waves(rng, axes, size, 0.6 * s0),
                    v0=_waves(rng, axes, size, 0.6 * s0 * 3000.0), notches=(v1, v2, p0),
                    bcs=[(2, 1, pulled, load)], bc=("add_y", pulled, load))


def _packing(case, rng):
    grid = (case["nx"], case["ny"], case["nz"])
    if case["layout"] == "settled":
        spacing, jitter, radii, speed = 2e-3 - 3e-7, 1e-7, (0.9999e-3, 1.0001e-3), 0.02
    else:
        spacing, jitter, radii, speed = 2.5e-3, 1.4e-4, (0.9e-3, 1.1e-3), 0.1
    axes, h = _grid(*grid, [spacing * n for n in grid])
    x = _points(axes)
    n = x.shape[0]
    x += rng.uniform(-jitter, jitter, (n, 3))
    radius = rng.uniform(*radii, n)
    params = dict(pd_model=0, contact_model=1, contact_radius=1.1e-3, radius_extend=0.22e-3,
                  nu=0.3, E=70e9, restitution=0.8, dt=1e-7, rebuild_every=10,
                  per_particle_radius=1)
    return _problem(params, x, grid, h, 4.0 / 3.0 * math.pi * radius ** 3, 2500.0, radius=radius,
                    v0=speed * rng.standard_normal((n, 3), dtype=np.float32).astype(np.float64))


def _cylinder(case, rng):
    outer, inner, height = 0.025, 0.02, 0.1
    c = case["across"]
    grid = (c, c, 2 * c)
    size = [2 * outer, 2 * outer, height]
    axes, h = _grid(*grid, size)
    x = _points(axes)
    r2 = x[:, 0] ** 2 + x[:, 1] ** 2
    cell = np.nonzero((r2 >= inner * inner) & (r2 <= outer * outer))[0]
    x = x[cell] + (rng.random((len(cell), 3)) - 0.5) * h
    K, sc, horizon = 130e9, 0.02, 4.17462 * h[0]
    zf = x[:, 2] / (0.5 * height)
    vr, ang = 200.0 - 50.0 * zf * zf, np.arctan2(x[:, 1], x[:, 0])
    v0 = np.stack([vr * np.cos(ang), vr * np.sin(ang), 100.0 * zf], 1)
    params = dict(pd_model=PMB, fracture=1, horizon=horizon, K=K,
                  G0=9 * K * horizon * sc * sc / 5, dt=1.7e-4 * h[0], contact_model=2,
                  contact_horizon=horizon, contact_K=K, contact_radius=0.45 * h[0],
                  radius_extend=0.01 * h[0], rebuild_every=0)
    return _problem(params, x, grid, h, h[0] * h[1] * h[2], 7800.0, v0=v0, cell=cell)


def _batch_cases(case, seed):
    """The instances' own cases: sizes log-uniform up to `largest`."""
    rng = np.random.Generator(np.random.PCG64([seed, case["jobs"], case["largest"]]))
    shape = np.random.Generator(np.random.PCG64([case["jobs"], case["largest"]]))
    out = []
    for k in range(case["jobs"]):
        n = math.exp(shape.uniform(math.log(1e3), math.log(case["largest"])))
        one = dict(kind=("wave", "box", "plate", "box")[k % 4], precision=case["precision"])
        if one["kind"] == "wave":
            s = max(8, round(n ** (1 / 3)))
            one.update(nx=s, ny=s, nz=s)
        elif one["kind"] == "plate":
            a = max(16, round((n / (0.5 * 0.045)) ** (1 / 3)))
            one.update(layout="deck", horizon=3.01, nx=a, ny=max(8, a // 2),
                       nz=max(2, round(0.045 * a)))
        else:
            a = max(30, round((n / (0.4 * 0.02)) ** (1 / 3)))
            one.update(nx=a, ny=max(12, round(0.4 * a)), nz=max(2, round(0.02 * a)))
        out.append((one, int(rng.integers(1 << 30))))
    return out


# ---------------------------------------------------------------------------
# The measured passes.

class _DeviceField:
    """A system's field as it lies on the device, component-major (a tensor made
    from it keeps the system open)."""

    def __init__(self, system, field):
        self.system = system
        ptr, stride = system.device_field(field)
        vector = field in ("u", "v", "f")
        self.__cuda_array_interface__ = dict(
            shape=(3, system.n) if vector else (system.n,),
            strides=(8 * stride, 8) if vector else (8,), typestr="<f8", data=(ptr, False),
            version=3)


def _fields(system, names):
    return {f: torch.as_tensor(_DeviceField(system, f), device="cuda") for f in names}


def _names(prob, output):
    names = ["u", "v", "f"]
    if prob["params"]["pd_model"] == LPS:
        names.append("theta")
    if output:
        names += ["W", "phi"] if prob["params"]["fracture"] else ["W"]
    return names


def _open(case, prob):
    system = cabanapd_b200.System(prob["params"], precision=PRECISION[case["precision"]])
    return problems.setup(system, prob)


def prepare(case, seed):
    if case["kind"] == "job":
        return dict(case=case, prob=_body(case, seed))
    if case["kind"] == "batch":
        systems = []
        for one, s in _batch_cases(case, seed):
            systems.append(_open(one, _body(one, s)))
        batch = cabanapd_b200.Batch(systems, [1 << 30] * len(systems))
        return dict(case=case, batch=batch, systems=systems,
                    fields=[_fields(s, ["u", "v"]) for s in systems])
    prob = _body(case, seed)
    system = _open(case, prob)
    return dict(case=case, system=system, fields=_fields(system, _names(prob, case["output"])))


def run(state):
    case = state["case"]
    if case["kind"] == "job":
        system = _open(case, state["prob"])
        totals = [system.step_energy(10) for _ in range(case["steps"] // 10)]
        u = system.get("u")
        system.close()
        return dict(totals=np.array(totals), u=u)
    if case["kind"] == "batch":
        state["batch"].step(case["steps"])
        return state["fields"]
    if case["output"]:
        totals = state["system"].step_energy(case["steps"])
        return dict(state["fields"], totals=np.array(totals))
    state["system"].step(case["steps"])
    return state["fields"]


# ---------------------------------------------------------------------------
# What a pass cannot do without.

def _offsets(h, reach):
    """Grid offsets within `reach` (one of each opposite pair is not left out)."""
    r = [int(reach / d) for d in h]
    return [(a, b, c) for c in range(-r[2], r[2] + 1) for b in range(-r[1], r[1] + 1)
            for a in range(-r[0], r[0] + 1)
            if (a, b, c) != (0, 0, 0) and
            (a * h[0]) ** 2 + (b * h[1]) ** 2 + (c * h[2]) ** 2 <= reach * reach]


def work(case):
    """Per step each particle's displacement and velocity are read and written
    once (96 B), each bond's state once (1 bit), and each pair of particles
    takes about 40 operations (LPS: 20 more for the dilatation, contact 60)."""
    if case["kind"] == "batch":
        each = [work(dict(one, steps=case["steps"])) for one, _ in _batch_cases(case, 0)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    if case["kind"] == "cylinder":
        c = case["across"]
        n = math.pi * (0.5 ** 2 - 0.4 ** 2) * c * c * 2 * c
        pairs = n * 0.6 * 4.0 / 3.0 * math.pi * 4.17462 ** 3 / 2
        return {"bytes": case["steps"] * (96 * n + pairs / 4), "flops": case["steps"] * 40 * pairs}
    grid = (case["nx"], case["ny"], case["nz"])
    n = grid[0] * grid[1] * grid[2]
    if case["kind"] == "packing":
        pairs = 3 * n
        return {"bytes": case["steps"] * 96 * n, "flops": case["steps"] * 60 * pairs}
    if case["kind"] == "wave":
        h, reach = [1.0, 1.0, 1.0], 3.01
    elif case["kind"] == "box":
        h = [0.1 / grid[0], 0.04 / grid[1], 0.002 / grid[2]]
        reach = 3.01 * h[0]
    else:
        deck = case["layout"] == "deck"
        h = [0.2 / grid[0], 0.1 / grid[1], 0.009 / grid[2]] if deck else [1.0, 1.0, 1.0]
        reach = case["horizon"] * h[0]
    pairs = sum(max(0, grid[0] - abs(a)) * max(0, grid[1] - abs(b)) * max(0, grid[2] - abs(c))
                for a, b, c in _offsets(h, reach)) / 2
    fracture = case["kind"] != "wave"
    flops = 60 if case["kind"] == "box" else 40
    steps = case["steps"]
    extra = 0.0
    if case["kind"] == "job":  # the job's arrays in (x, u, v, vol, rho) and u out
        extra = n * (24 * 3 + 8 * 2 + 24)
    return {"bytes": steps * (96 * n + (pairs / 4 if fracture else 0)) + extra,
            "flops": steps * flops * pairs}


# ---------------------------------------------------------------------------
# The same physics in plain float64 torch.

class _Exact:
    """Velocity Verlet on a grid of cells; fields are [3][nz][ny][nx] (zero in
    cells without a particle), bonds a list of (offset, intact) pairs."""

    def __init__(self, prob):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        p = self.p = prob["params"]
        self.prob, self.grid, self.h = prob, prob["grid"], prob["h"]
        g = self.shape = tuple(reversed(self.grid))
        self.cells = None if prob["cell"] is None else self._t(prob["cell"])
        self.here = torch.zeros(g, dtype=torch.bool, device=self.dev)
        if self.cells is None:
            self.here[:] = True
        else:
            self.here.view(-1)[self.cells] = True
        self.x = self._vector(prob["x"])
        self.u, self.v = self._vector(prob["u0"]), self._vector(prob["v0"])
        self.vol, self.rho = self._scalar(prob["vol"]), self._scalar(prob["rho"])
        self.rho = torch.where(self.here, self.rho, torch.ones_like(self.rho))
        self.radius = self._scalar(prob["radius"])
        self.nofail = self._scalar(prob["nofail"]) != 0
        self.model, self.fracture = p["pd_model"], p.get("fracture", 0)
        self.theta = None
        if self.model:
            d = p["horizon"]
            self.c = 18.0 * p["K"] / (math.pi * d ** 4)
            if self.fracture:
                k = 8.0 / 15.0 if p.get("influence_type") == 0 else 5.0 / 9.0
                self.bbc = (1.0 + math.sqrt(k * p["G0"] / p["K"] / d)) ** 2
            if self.model == LPS:
                self.ct, self.cs = 3.0 * p["K"] - 5.0 * p["G"], 15.0 * p["G"]
            self._find_bonds(d + 1e-14)
        # Contact beside bonds acts from the first step on.
        self.f = self._forces(contact=not self.model)
        self._bc()

    def _t(self, a):
        return torch.as_tensor(np.ascontiguousarray(a)).to(self.dev)

    def _scalar(self, a):
        out = torch.zeros(self.shape, dtype=torch.float64, device=self.dev)
        if a is not None:
            a = self._t(a).double()
            if self.cells is None:
                out.view(-1)[:] = a
            else:
                out.view(-1)[self.cells] = a
        return out

    def _vector(self, a):
        return torch.stack([self._scalar(None if a is None else a[:, d]) for d in range(3)])

    def out(self, a):
        """A field in the particles' order."""
        a = a.reshape(3, -1) if a.dim() == 4 else a.reshape(-1)
        return a if self.cells is None else a[..., self.cells]

    def _cut(self, o):
        """Slices (last three axes) of the rows with a neighbour at offset o, and of it."""
        me, other = [], []
        for n, d in zip(self.shape, reversed(o)):
            me.append(slice(max(0, -d), n - max(0, d)))
            other.append(slice(max(0, d), n + min(0, d)))
        return (...,) + tuple(me), (...,) + tuple(other)

    def _find_bonds(self, reach):
        # Particles may sit anywhere in their cell: one cell further on each side.
        wide = 1.0 + 1e-9 if self.cells is None else 1.0 + 1.8 / 4.0
        self.bonds = []
        notch = self.prob["notches"]
        for o in _offsets(self.h, reach * wide):
            if any(abs(d) >= n for d, n in zip(o, self.grid)):
                continue
            a, b = self._cut(o)
            xi = self.x[b] - self.x[a]
            on = (xi * xi).sum(0) <= reach * reach
            if self.cells is not None:
                on &= self.here[a] & self.here[b]
            if not bool(on.any()):
                continue
            whole = on.clone()
            if notch is not None:
                for v1, v2, p0 in zip(*notch):
                    on &= ~_crosses(v1, v2, p0, self.x[a], xi)
            self.bonds.append((o, on, whole))

    def _pair(self, o):
        a, b = self._cut(o)
        xi = self.x[b] - self.x[a]
        eta = self.u[b] - self.u[a]
        r = xi + eta
        l2 = (xi * xi).sum(0)
        xil = l2.sqrt()
        rl = (r * r).sum(0).sqrt()
        if self.cells is not None:
            xil, rl = xil.clamp_min(1e-30), rl.clamp_min(1e-30)
        s = (eta * (2.0 * xi + eta)).sum(0) / (xil * (rl + xil))
        return a, b, r, rl, xil, s

    def _forces(self, contact=True):
        f = torch.zeros_like(self.u)
        if self.model == LPS:
            m, th = torch.zeros_like(self.vol), torch.zeros_like(self.vol)
            for o, on, _ in self.bonds:
                a, b, r, rl, xil, s = self._pair(o)
                w = on * xil * xil * self.vol[b]
                m[a] += w
                th[a] += w * s
            self.m, self.theta = m, torch.where(m > 0, 3.0 * th / m, torch.zeros_like(m))
        if self.model:
            for o, on, _ in self.bonds:
                a, b, r, rl, xil, s = self._pair(o)
                if self.fracture:
                    safe = self.nofail[a] if self.model == LPS else self.nofail[a] | self.nofail[b]
                    on &= ~((rl * rl >= self.bbc * xil * xil) & ~safe)
                if self.model == LPS:
                    k = (self.ct * (self.theta[a] / self.m[a] + self.theta[b] / self.m[b]) +
                         s * (self.cs / self.m[a] + self.cs / self.m[b])) * xil
                else:
                    k = self.c * s
                f[a] += torch.where(on, k * self.vol[b] / rl, torch.zeros_like(k)) * r
        if contact and self.p.get("contact_model", 0):
            self._contact(f)
        return f

    def _contact(self, f):
        p = self.p
        hertz = p["contact_model"] == 1
        # Spheres meet only the face neighbours of their own cell; the cylinder's
        # particles any within a contact radius.
        for o in _offsets(self.h, 1.01 * self.h[0] if hertz else 2.9 * self.h[0]):
            a, b, r, rl, _, _ = self._pair(o)
            n = r / rl
            if hertz:
                es = p["E"] / (2.0 * (1.0 - p["nu"] ** 2))
                lne = math.log(p["restitution"])
                damp = 2.0 * math.sqrt(5.0 / 6.0) * -lne / math.sqrt(lne * lne + math.pi ** 2)
                vn = ((self.v[b] - self.v[a]) * n).sum(0)
                ra, rb = self.radius[a], self.radius[b]
                over = (ra + rb - rl).clamp_min(0.0)
                rs = ra * rb / (ra + rb)
                ma, mb = self.rho[a] * self.vol[a], self.rho[b] * self.vol[b]
                ms = ma * mb / (ma + mb)
                k = -4.0 / 3.0 * es * rs.sqrt() * over ** 1.5
                k = k + damp * (2.0 * es * (rs * over).sqrt() * ms).sqrt() * vn
                k = k / self.vol[a]
            else:
                c = 18.0 * p["contact_K"] / (math.pi * p["contact_horizon"] ** 4)
                rc = p["contact_radius"]
                near = (rl < rc) & self.here[a] & self.here[b]
                k = torch.where(near, 15.0 * c * (rl - rc) / p["contact_horizon"] * self.vol[b],
                                torch.zeros_like(rl))
            f[a] += k * n

    def _bc(self):
        if self.prob["bc"] is None:
            return
        kind, rows, values = self.prob["bc"]
        rows = self._t(rows)
        if kind == "zero":
            self.f.view(3, -1)[:, rows] = 0.0
        else:
            self.f.view(3, -1)[1, rows] += self._t(values)

    def step(self, n):
        dt = self.p["dt"]
        for _ in range(n):
            self.v += 0.5 * dt / self.rho * self.f
            self.u += dt * self.v
            self.f = self._forces()
            self._bc()
            self.v += 0.5 * dt / self.rho * self.f

    def energy(self):
        """W per particle, damage per particle (or None), totals."""
        W, left, all_ = (torch.zeros_like(self.vol) for _ in range(3))
        if self.model == LPS:
            W += 0.5 * self.ct / 3.0 * self.theta ** 2
        for o, on, whole in self.bonds:
            a, b, r, rl, xil, s = self._pair(o)
            vb = self.vol[b]
            if self.model == LPS:
                W[a] += on * (0.5 * self.cs / self.m[a] * s * s * xil * xil * vb)
            else:
                W[a] += on * (0.25 * self.c * s * s * xil * vb)
            left[a] += on * vb
            all_[a] += whole * vb
        phi = 1.0 - left / all_ if self.fracture else None
        return W, phi, [float((W * self.vol).sum()), float(phi.sum()) if self.fracture else 0.0]


def _crosses(v1, v2, p0, x, l):
    """Whether the bonds from x along l cross the parallelogram p0 + a v1 + b v2
    (bonds parallel to its plane: within the plane and overlapping it)."""
    cv = np.cross(v1, v2)
    n2 = float(cv @ cv)
    n = cv / math.sqrt(n2)
    dot = lambda w, a: w[0] * a[0] + w[1] * a[1] + w[2] * a[2]  # noqa: E731
    rel = [x[d] - float(p0[d]) for d in range(3)]
    ln = dot(l, n)
    dist = -dot(rel, n)
    flat = ln.abs() < 1e-10
    in_plane = flat & (dist.abs() < 1e-10)
    t = dist / torch.where(flat, torch.ones_like(ln), ln)
    # (w x v2) . cv = w . (v2 x cv)
    e1, e2 = np.cross(v2, cv) / n2, -np.cross(v1, cv) / n2
    hit = [rel[d] + t * l[d] for d in range(3)]
    a, b, tol = dot(hit, e1), dot(hit, e2), 1e-10
    cut = (~flat & (t > -tol) & (t < 1 + tol) & (torch.minimum(a, b) > -tol) &
           (torch.maximum(a, b) < 1 + tol))
    if bool(in_plane.any()):
        end = [rel[d] + l[d] for d in range(3)]
        apart = torch.zeros_like(cut)
        for e in (e1, e2):
            i, j = dot(rel, e), dot(end, e)
            apart |= (torch.minimum(i, j) > 1 + tol) | (torch.maximum(i, j) < -tol)
        cut |= in_plane & ~apart
    return cut


def exact(case, seed):
    if case["kind"] == "batch":
        out = []
        for one, s in _batch_cases(case, seed):
            e = _Exact(_body(one, s))
            e.step(case["steps"])
            out.append(dict(u=e.out(e.u), v=e.out(e.v)))
        return out
    prob = _body(case, seed)
    e = _Exact(prob)
    if case["kind"] == "job":
        totals = []
        for _ in range(case["steps"] // 10):
            e.step(10)
            totals.append(e.energy()[2])
        return dict(totals=np.array(totals), u=e.out(e.u).T)
    e.step(case["steps"])
    out = {f: e.out(getattr(e, f)) for f in _names(prob, False)}
    if case["output"]:
        W, phi, totals = e.energy()
        out["W"] = e.out(W)
        if phi is not None:
            out["phi"] = e.out(phi)
        out["totals"] = np.array(totals)
    return out
