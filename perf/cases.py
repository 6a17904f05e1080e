"""The work a user has this framework do, as cases that can be timed.

Kinds of case, each through the public entry points:

* ``run``           one TrajectorySimulator.run_simulation call: molecules drawn on the device, counts back
* ``batch``         one run_simulations call over many batches of molecules
* ``outputs``       Engine.run on initial conditions in device memory, per-molecule results to device tensors
* ``trajectories``  run_simulation with apertures of interest: the kept molecules' full trajectories
* ``sweep``         one run_sweep call over lens voltages x Stark tables
* ``gradient``      soft_loss forward and backward: the soft transmission and its six parameter gradients

Beamlines: ``lens`` is the benchmark's hexapole lens beamline (states the lens defocuses, "high", or focuses,
"low", with a 10 mm detector), ``ballistic`` its three-aperture beamline, ``example`` the lens beamline of the
reference's example scripts (disc source, radial force table, dz = 1 mm, field plates).
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
if str(ROOT / "centrex-molecule-trajectories_gb300") not in sys.path:
    sys.path.insert(0, str(ROOT / "centrex-molecule-trajectories_gb300"))

import ctraj  # noqa: E402
from ctraj.adjoint import SoftProblem, soft_loss  # noqa: E402
from ctraj.compiler import compile_beamline  # noqa: E402
from ctraj.engine import default_engine  # noqa: E402
from ctraj.sweep import run_sweep  # noqa: E402
from ctraj.workloads import ballistic_beamline, lens_beamline, source, sweep_configs  # noqa: E402

G = 9.80665


def listed():
    return [
        # a quick look at a beamline: launches and the slowest molecule's chain of steps are all there is
        dict(name="lens_1e4", kind="run", beamline="lens", seeker="high", n=10_000, precision=32),
        # the ordinary size of the example scripts, in the state the lens focuses: most entrants stay to its end
        dict(name="lens_focus_1e6", kind="run", beamline="lens", seeker="low", n=1_000_000, precision=32),
        # the benchmark's beamline and size, one run at a time
        dict(name="lens_1e7", kind="run", beamline="lens", seeker="high", n=10_000_000, precision=32),
        # the example scripts' beamline with its disc source, radial table and 1 mm steps
        dict(name="example_1e6", kind="run", beamline="example", seeker="high", n=1_000_000, precision=32),
        # the exact mode, used to check the fast one: the reference's own arithmetic through the lens
        dict(name="lens_fp64_1e5", kind="run", beamline="lens", seeker="high", n=100_000, precision=64),
        # the benchmark's loop of runs as one call: throughput
        dict(name="batch_20x1e7", kind="batch", beamline="lens", seeker="high", n=10_000_000, runs=20),
        # the ballistic workload in the exact mode, every molecule's label and last row kept on the device
        dict(name="ballistic_fp64_1e5", kind="outputs", beamline="ballistic", seeker="high", n=100_000, precision=64),
        # the same for the lens beamline in the fast mode: a caller that studies losses molecule by molecule
        dict(name="lens_outputs_1e6", kind="outputs", beamline="lens", seeker="high", n=1_000_000, precision=32),
        # the trajectories of the detected molecules, what the reference's users plot
        dict(name="trajectories_1e6", kind="trajectories", beamline="example", seeker="high", n=1_000_000, precision=32),
        # a voltage scan over four states: a quarter of the benchmark's voltages, its molecules per configuration
        dict(name="sweep_64x4", kind="sweep", voltages=64, n_min=10_000, n_max=1_000_000),
        # one step of tuning a beamline by gradient descent, at the benchmark's size
        dict(name="gradient_1e6", kind="gradient", seeker="low", n=1_000_000, precision=32, drawn=True),
        # the check of a gradient in 64 bits on given normals
        dict(name="gradient_fp64_1e4", kind="gradient", seeker="low", n=10_000, precision=64, drawn=False),
    ]


def draw(rng):
    def size(lo, hi):  # spread over the logarithm, mostly odd, in the hundreds that run_simulation takes
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | 1

    kind = rng.choice(["run", "run", "run", "batch", "outputs", "trajectories", "sweep", "gradient"])
    seeker = rng.choice(["high", "low"])
    beamline = rng.choice(["lens", "lens", "example"])
    if kind == "run":
        precision = rng.choice([32, 32, 64])
        return dict(kind=kind, beamline=beamline, seeker=seeker, precision=precision,
                    n=size(3_000, 20_000_000 if precision == 32 else 500_000))
    if kind == "batch":
        runs = rng.randrange(2, 25)
        return dict(kind=kind, beamline=beamline, seeker="high", runs=runs, n=size(30_000, 100_000_000 / runs))
    if kind == "outputs":
        precision = rng.choice([32, 64])
        beamline = rng.choice(["lens", "ballistic"])
        return dict(kind=kind, beamline=beamline, seeker="high", precision=precision,
                    n=size(3_000, 100_000 if precision == 64 and beamline == "lens" else 1_000_000))
    if kind == "trajectories":
        return dict(kind=kind, beamline="example", seeker="high", precision=rng.choice([32, 64]), n=size(30_000, 1_000_000))
    if kind == "sweep":
        return dict(kind=kind, voltages=rng.randrange(3, 80), n_min=size(1_000, 20_000), n_max=size(50_000, 800_000))
    precision = rng.choice([32, 32, 64])
    return dict(kind=kind, seeker=seeker, precision=precision, drawn=rng.random() < 0.6,
                n=size(3_000, 3_000_000 if precision == 32 else 20_000))


# ---------------------------------------------------------------------------
# what a user's program has in hand
# ---------------------------------------------------------------------------

def _example_beamline():
    """The example scripts' lens beamline, its force table built the reference's way from a two-level Stark
    curve (the TlF curve needs a package that is not here), in the state the lens focuses."""
    W = ctraj.TwoLevelStark(6.7e9, 4.2, 1.0)
    inch = 0.0254
    lens = ctraj.ElectrostaticLens(name="ES lens", z0=1.00838, L=0.6,
                                   a_interp=ctraj.reference_radial_table(W, V=27.6e3, d=1.75 * inch))
    return ctraj.Beamline([
        ctraj.CircularAperture(name="4K shield", z0=1.7 * inch, L=0.25 * inch, d=1 * inch),
        ctraj.CircularAperture(name="40K shield", z0=3.2 * inch, L=0.25 * inch, d=1 * inch),
        ctraj.CircularAperture(name="BB exit", z0=5.95 * inch, L=0.75 * inch, d=4 * inch),
        lens,
        ctraj.FieldPlates(name="Field plates", z0=2.43, L=3.0, w=0.02),
        ctraj.RectangularAperture(name="DR aperture", z0=6.44346, L=0.25 * inch, w=0.018, h=0.03),
    ])


_beamlines = {}


def _beamline(case):
    """(beamline, xdist, vdist); a program builds its beamline once and runs it many times."""
    which = case.get("beamline", "lens")
    key = (which, case.get("seeker"))
    if key not in _beamlines:
        if which == "example":
            _beamlines[key] = (_example_beamline(), ctraj.CeNTREXPositionDistribution(), ctraj.CeNTREXVelocityDistribution())
        elif which == "ballistic":
            _beamlines[key] = (ballistic_beamline(), *source())
        elif case["seeker"] == "low":
            _beamlines[key] = (lens_beamline(V=10e3, low_field_seeker=True, detector_d=10e-3), *source())
        else:
            _beamlines[key] = (lens_beamline(), *source())
    return _beamlines[key]


def _initial_conditions(n, seed):
    """(6, n) float64: the workloads' Gaussian source."""
    g = np.random.default_rng(seed)
    ics = g.standard_normal((6, n)) * np.array([1.5e-3, 1.5e-3, 0.0, 20.0, 20.0, 16.0])[:, None]
    ics[5] += 184.0
    return ics


def _normals(n, seed):
    return np.random.default_rng(seed).standard_normal((5, n))


def _params(prob, seed):
    """A point of a tuning run near the design: every parameter moved by up to 2 %."""
    return prob.initial_params() * (1 + 0.02 * np.random.default_rng(seed + 1).uniform(-1, 1, 6))


def _soft_problem(case, seed):
    bl, xd, vd = _beamline(case)
    kw = {} if case["drawn"] else dict(normals=_normals(case["n"], seed))
    return SoftProblem.from_beamline(bl, n=case["n"], xdist=xd, vdist=vd, aperture="A1", precision=case["precision"],
                                     seed=seed, **kw)


def prepare(case, seed):
    kind, n = case["kind"], case.get("n")
    s = dict(case=case, seed=seed, kind=kind)
    if kind in ("run", "batch", "trajectories"):
        s["sim"] = ctraj.TrajectorySimulator(precision=case.get("precision", 32))
        s["beamline"], s["xdist"], s["vdist"] = _beamline(case)
    elif kind == "outputs":
        s["cb"] = compile_beamline(_beamline(case)[0])
        s["ics"] = torch.as_tensor(_initial_conditions(n, seed), device="cuda")
        s["out"] = dict(label=torch.empty(n, dtype=torch.int32, device="cuda"),
                        rows=torch.empty(n, dtype=torch.int32, device="cuda"),
                        margin=torch.empty(n, dtype=torch.float64, device="cuda"),
                        final=torch.empty((10, n), dtype=torch.float64, device="cuda"))
    elif kind == "sweep":
        s["beamline"], s["xdist"], s["vdist"] = _beamline(dict(beamline="lens", seeker="high"))
        s["configs"] = sweep_configs(n_voltages=case["voltages"], n_min=case["n_min"], n_max=case["n_max"], seed=seed)
    else:
        s["prob"] = _soft_problem(case, seed)
        s["params"] = torch.tensor(_params(s["prob"], seed), dtype=torch.float64, requires_grad=True)
    return s


def _padded(trajectories, n):
    """The trajectories as one array (molecules, rows, 10), NaN where there is none: one shape for every seed."""
    out = np.full((n // 10_000 + 32, 640, 10), np.nan)
    for k, t in enumerate(trajectories):
        o = out[k, :t.n]
        o[:, :3], o[:, 3:6], o[:, 6:9], o[:, 9] = t.x, t.v, t.a, t.t
    return out


def run(s):
    case, kind = s["case"], s["kind"]
    if kind == "run":
        sim = s["sim"]
        sim.run_simulation(s["beamline"], "run", s["vdist"], s["xdist"], N_traj=case["n"], seed=s["seed"])
        return dict(counts=sim.last_run.counts, steps=sim.last_run.molecule_steps)
    if kind == "batch":
        sim, k = s["sim"], case["runs"]
        names = [f"batch{j}" for j in range(k)]
        sim.run_simulations(s["beamline"], names, s["vdist"], s["xdist"], N_traj=case["n"],
                            seeds=range(s["seed"] * 1000, s["seed"] * 1000 + k))
        return dict(counts=np.stack([r.counts for r in sim.last_runs]),
                    steps=np.array([r.molecule_steps for r in sim.last_runs]))
    if kind == "outputs":
        r = default_engine().run(s["cb"], case["n"], precision=case["precision"], ics=s["ics"], device_outputs=s["out"])
        return dict(s["out"], counts=r.counts, steps=r.molecule_steps)
    if kind == "trajectories":
        sim = s["sim"]
        sim.run_simulation(s["beamline"], "run", s["vdist"], s["xdist"], N_traj=case["n"],
                           apertures_of_interest=["Detected"], seed=s["seed"])
        return dict(counts=sim.last_run.counts, rows=_padded([m.trajectory for m in sim.result.molecules], case["n"]))
    if kind == "sweep":
        r = run_sweep(s["beamline"], s["configs"], s["xdist"], s["vdist"], seed=s["seed"])
        return dict(counts=r.counts, totals=r.totals, steps=r.molecule_steps)
    p = s["params"]
    p.grad = None
    loss = soft_loss(p, s["prob"])
    loss.backward()
    return dict(loss=loss.detach(), grad=p.grad)


def work(case):
    """Floating-point operations: 114 per RK4 step (four table-driven forces of 14, the stage points, the
    combination), 12 per ballistic flight, 60 for a molecule's draw; RK4 steps per molecule as these beamlines
    give them.  Bytes: initial conditions read, results written."""
    kind = case["kind"]
    rk4 = {("lens", "high"): 14.3, ("lens", "low"): 56.0, ("example", "high"): 2.4, ("ballistic", "high"): 0.0}
    per = lambda c: 114 * rk4[(c.get("beamline", "lens"), "high" if c.get("beamline", "lens") != "lens"  # noqa: E731
                               else c["seeker"])] + 12 * 1.1 + 60
    if kind == "run":
        return dict(bytes=64, flops=case["n"] * per(case))
    if kind == "batch":
        return dict(bytes=64 * case["runs"], flops=case["runs"] * case["n"] * per(case))
    if kind == "outputs":
        return dict(bytes=case["n"] * (6 * 8 + 4 + 4 + 8 + 80), flops=case["n"] * per(case))
    if kind == "trajectories":  # about one molecule in 30000 is detected, with 613 rows of ten values
        return dict(bytes=case["n"] / 30000 * 613 * 80, flops=case["n"] * per(case))
    if kind == "sweep":
        lo, hi = case["n_min"], case["n_max"]
        n = 4 * case["voltages"] * ((hi - lo) / math.log(hi / lo) if hi > lo else lo)
        return dict(bytes=4 * case["voltages"] * 40, flops=n * (114 * 22.5 + 12 * 1.1 + 60))
    # gradient: the soft forward pass and, for the survivors, its recomputation and the transposed steps
    return dict(bytes=64 + (0 if case["drawn"] else case["n"] * 40), flops=case["n"] * 3 * per(case))


# ---------------------------------------------------------------------------
# the same results in 64 bits: plain numpy, no code of the package (its objects are read as data)
# ---------------------------------------------------------------------------

def _philox_words(n, seed):
    """Words w0..w7 of molecules 0..n-1: Philox-4x32-10 (Salmon et al. 2011), key = seed, counter = (i, call)."""
    out = []
    lo32 = np.uint64(0xFFFFFFFF)
    for call in (0, 1):
        c0, c1 = np.arange(n, dtype=np.uint64), np.zeros(n, np.uint64)
        c2, c3 = np.full(n, call, np.uint64), np.zeros(n, np.uint64)
        k0, k1 = seed & 0xFFFFFFFF, seed >> 32
        for _ in range(10):
            p0, p1 = np.uint64(0xD2511F53) * c0, np.uint64(0xCD9E8D57) * c2
            c0, c1, c2, c3 = (p1 >> np.uint64(32)) ^ c1 ^ np.uint64(k0), p1 & lo32, \
                (p0 >> np.uint64(32)) ^ c3 ^ np.uint64(k1), p0 & lo32
            k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
        out += [c0, c1, c2, c3]
    return out


def _drawn_ics(n, seed, xd, vd):
    """Initial conditions of a disc source: Box-Muller normals for the velocity, (angle, radius) for the position."""
    u = [(w.astype(np.float64) + 0.5) * 2.0 ** -32 for w in _philox_words(n, seed)]
    r = [np.sqrt(-2 * np.log(u[k])) for k in (0, 2)]
    v = (vd.vx + vd.sigmax * r[0] * np.cos(2 * np.pi * u[1]), vd.vy + vd.sigmay * r[0] * np.sin(2 * np.pi * u[1]),
         vd.vz + vd.sigmaz * r[1] * np.cos(2 * np.pi * u[3]))
    rho = np.sqrt(u[7]) * xd.d / 2
    return np.stack([rho * np.cos(2 * np.pi * u[6]), rho * np.sin(2 * np.pi * u[6]), np.full(n, xd.z), *v])


def _acceleration(lens, x, y):
    f = lens.a_interp
    r = np.hypot(x, y)
    if hasattr(f, "coef"):
        E = f.alpha * r * r
        j = np.clip(((E - f.knots[0]) / (f.knots[1] - f.knots[0])).astype(np.int64), 0, len(f.knots) - 2)
        s, c = E - f.knots[j], f.coef[j]
        w = -(c[:, 2] + s * (2 * c[:, 1] + s * 3 * c[:, 0])) * 2 * f.alpha / f.mass
    else:
        w = np.interp(r, f.x, f.y) / np.where(r > 0, r, 1)
    return w * x, w * y - G


class _Walk:
    """Molecules through a beamline with the reference's rules, in float64 numpy."""

    def __init__(self, ics, keep_rows=False):
        n = ics.shape[1]
        self.S = np.concatenate([ics, np.zeros((4, n))])  # x y z vx vy vz ax ay az t
        self.S[7] = -G
        self.margin = np.full(n, np.inf)
        self.alive = np.arange(n)
        self.trace = [[(np.arange(n), self.S.copy())]] if keep_rows else None

    def store(self, i):
        if self.trace is not None:
            self.trace[0].append((i, self.S[:, i].copy()))

    def fly(self, z, dt=None, i=None):
        i = self.alive if i is None else i
        S = self.S[:, i]
        dt = (z - S[2]) / S[5] if dt is None else dt
        for k in range(3):
            S[k] = S[k] + S[3 + k] * dt + S[6 + k] * dt * dt / 2
            S[3 + k] = S[3 + k] + S[6 + k] * dt
        S[9] += dt
        S[6], S[7], S[8] = 0.0, -G, 0.0
        self.S[:, i] = S
        self.store(i)

    def note(self, i, *dist):
        for d in dist:
            self.margin[i] = np.minimum(self.margin[i], np.abs(d))

    def circle(self, R):
        i = self.alive
        d = np.hypot(self.S[0, i], self.S[1, i]) - R
        self.note(i, d)
        self.alive = i[d <= 0]

    def walk(self, elements):
        for e in elements:
            kind = type(e).__name__
            self.fly(e.z0)
            if kind == "ElectrostaticLens":
                self.circle(e.d / 2)
                self.lens(e)
            elif kind == "CircularAperture":
                self.circle(e.d / 2)
                self.fly(e.z1)
                self.circle(e.d / 2)
            elif kind == "RectangularAperture":
                for z in (None, e.z1):
                    if z is not None:
                        self.fly(z)
                    i = self.alive
                    x, y = self.S[0, i], self.S[1, i]
                    self.note(i, x - e.x1, x - e.x2, y - e.y1, y - e.y2)
                    self.alive = i[(e.x1 < x) & (x < e.x2) & (e.y1 < y) & (y < e.y2)]
            else:  # field plates
                i = self.alive
                x = self.S[0, i]
                self.note(i, x - e.x1, x - e.x2)
                i = i[(e.x1 < x) & (x < e.x2)]
                S = self.S[:, i]
                xe = S[0] + S[3] * (e.z1 - S[2]) / S[5]
                self.note(i, xe - e.x1, xe - e.x2)
                hit = ~((e.x1 < xe) & (xe < e.x2))
                h = i[hit]
                vx = self.S[3, h]
                self.fly(None, (np.where(vx < 0, e.x1, e.x2) - self.S[0, h]) / vx, h)
                self.alive = i[~hit]
                self.fly(e.z1)

    def lens(self, e):
        i = self.alive
        vz = self.S[5, i]
        dz = vz * e.dt if e.dt is not None else np.full(i.size, e.dz)
        N, dt = np.rint(e.L / dz).astype(np.int64), dz / vz
        out = [i[N == 0]]
        act, k = N > 0, 0
        i, N, dt = i[act], N[act], dt[act]
        while i.size:
            S = self.S[:, i]
            x, y, vx, vy = S[0], S[1], S[3], S[4]
            a1 = _acceleration(e, x, y)
            a2 = _acceleration(e, x + dt * vx, y + dt * vy)
            a3 = _acceleration(e, x + dt / 2 * (vx + dt / 2 * a1[0]), y + dt / 2 * (vy + dt / 2 * a1[1]))
            a4 = _acceleration(e, x + dt * (vx + dt / 2 * a2[0]), y + dt * (vy + dt / 2 * a2[1]))
            for c, v in ((0, vx), (1, vy)):
                S[c] = S[c] + dt * v + dt * dt / 6 * (a1[c] + a2[c] + a3[c])
                S[3 + c] = v + dt / 6 * (a1[c] + 2 * a2[c] + 2 * a3[c] + a4[c])
                S[6 + c] = a1[c]
            S[2] += dt * S[5]
            S[9] += dt
            self.S[:, i] = S
            self.store(i)
            k += 1
            d = np.hypot(S[0], S[1]) - e.d / 2
            self.note(i, d)
            on, end = d <= 0, N == k
            out.append(i[on & end])
            on &= ~end
            i, N, dt = i[on], N[on], dt[on]
        self.alive = np.sort(np.concatenate(out))
        self.fly(e.z1)


def _exact_soft(case, seed):
    """Loss and gradient of the soft transmission: forward-mode derivatives carried beside each value, as arrays
    (5, molecules) of (value, d/dV, d/dz0, d/dsigma_vx, d/dsigma_vy); the radii's enter only the edge weights."""
    bl, xd, vd = _beamline(case)
    els = bl.elements
    li = [type(e).__name__ for e in els].index("ElectrostaticLens")
    lens, f = els[li], els[li].a_interp
    r_a1 = els[0].d / 2
    p = np.array([f.V, lens.z0, r_a1, lens.d / 2, vd.sigmax, vd.sigmay]) * \
        (1 + 0.02 * np.random.default_rng(seed + 1).uniform(-1, 1, 6))
    V, z0, r_a1, bore = p[:4]
    nrm = _normals(case["n"], seed)

    def const(v, slot=None, d=1.0):
        o = np.zeros((5, np.size(v)))
        o[0] = v
        if slot is not None:
            o[slot] = d
        return o

    def mul(a, b):
        o = a[:1] * b + a * b[:1]
        o[0] = a[0] * b[0]
        return o

    vz = vd.vz + vd.sigmaz * nrm[2]
    x, y = const(xd.sigmax * nrm[3]), const(xd.sigmay * nrm[4])
    vx, vy = const(vd.vx + p[4] * nrm[0], 3, nrm[0]), const(vd.vy + p[5] * nrm[1], 4, nrm[1])
    lw, d_ap, d_bore = np.zeros((5, case["n"])), np.zeros(case["n"]), np.zeros(case["n"])

    def edge(x, y, R, on=None):
        """log sigma((R - r) / w) and d / dR."""
        r = np.hypot(x[0], y[0])
        dr = (x[0] * x + y[0] * y) / np.where(r > 0, r, 1)
        z = (R - r) / 0.2e-3
        e = np.exp(-np.abs(z))
        dls = np.where(z >= 0, e, 1) / (1 + e) / 0.2e-3
        ls = -dls * dr
        ls[0] = np.minimum(z, 0) - np.log1p(e)
        return (ls, dls) if on is None else (np.where(on, ls, 0), np.where(on, dls, 0))

    def fly(x, y, vx, vy, t):
        g = const(np.full(t.shape[1], -G))
        h = mul(t, t) / 2
        return x + mul(vx, t), y + mul(vy, t) + mul(g, h), vy + mul(g, t)

    z = xd.z
    for e in els[:li]:
        for zp in (e.z0, e.z1):
            x, y, vy = fly(x, y, vx, vy, const((zp - z) / vz))
            z = zp
            ls, d = edge(x, y, r_a1)
            lw, d_ap = lw + ls, d_ap + d
    x, y, vy = fly(x, y, vx, vy, const((z0 - z) / vz, 2, 1 / vz))
    ls, d = edge(x, y, bore)
    lw, d_bore = lw + ls, d_bore + d
    k = np.flatnonzero(lw[0] >= -30)
    x, y, vx, vy, lw, vz, d_ap, d_bore = x[:, k], y[:, k], vx[:, k], vy[:, k], lw[:, k], vz[k], d_ap[k], d_bore[k]
    N = np.rint(lens.L / (vz * lens.dt)).astype(np.int64)
    dt = lens.dt
    alpha, h = 3 * V / f.R ** 3, f.knots[1] - f.knots[0]

    def accel(x, y):
        r2 = mul(x, x) + mul(y, y)
        s = alpha * r2[0] - f.knots[0]
        j = np.clip((s / h).astype(np.int64), 0, len(f.knots) - 2)
        u, c = s - (f.knots[j] - f.knots[0]), f.coef[j]
        P, dP = c[:, 2] + u * (2 * c[:, 1] + u * 3 * c[:, 0]), 2 * c[:, 1] + u * 6 * c[:, 0]
        w = (dP * alpha) * r2  # d W'(E) by r^2; V enters through alpha as well
        w[0] = P
        w[1] += dP * r2[0] * alpha / V
        w *= -2 * alpha / f.mass
        w[1] += w[0] / V
        ay = mul(w, y)
        ay[0] -= G
        return mul(w, x), ay

    for step in range(int(N.max(initial=0))):
        on = step < N
        a1 = accel(x, y)
        a2 = accel(x + dt * vx, y + dt * vy)
        a3 = accel(x + dt / 2 * (vx + dt / 2 * a1[0]), y + dt / 2 * (vy + dt / 2 * a1[1]))
        a4 = accel(x + dt * (vx + dt / 2 * a2[0]), y + dt * (vy + dt / 2 * a2[1]))
        nx = x + dt * vx + dt * dt / 6 * (a1[0] + a2[0] + a3[0])
        ny = y + dt * vy + dt * dt / 6 * (a1[1] + a2[1] + a3[1])
        vx = np.where(on, vx + dt / 6 * (a1[0] + 2 * a2[0] + 2 * a3[0] + a4[0]), vx)
        vy = np.where(on, vy + dt / 6 * (a1[1] + 2 * a2[1] + 2 * a3[1] + a4[1]), vy)
        x, y = np.where(on, nx, x), np.where(on, ny, y)
        ls, d = edge(x, y, bore, on)
        lw, d_bore = lw + ls, d_bore + d
        if step % 256 == 255:  # the weightless go
            k = np.flatnonzero(lw[0] >= -60)
            x, y, vx, vy, lw = x[:, k], y[:, k], vx[:, k], vy[:, k], lw[:, k]
            vz, d_ap, d_bore, N = vz[k], d_ap[k], d_bore[k], N[k]
    for e in els[li + 1:]:
        for zp in (e.z0, e.z1):
            if math.isfinite(e.d):
                px, py, _ = fly(x, y, vx, vy, const((zp - z0 - N * vz * lens.dt) / vz, 2, -1 / vz))
                lw = lw + edge(px, py, e.d / 2)[0]
    w = np.exp(lw[0]) * (lw[0] >= -30)
    n = case["n"]
    grad = [w @ lw[1], w @ lw[2], w @ d_ap, w @ d_bore, w @ lw[3], w @ lw[4]]
    return dict(loss=np.array(w.sum() / n), grad=np.array(grad) / n)


def exact(case, seed):
    kind = case["kind"]
    if kind == "gradient" and not case["drawn"] and case["n"] <= 50_000:
        return _exact_soft(case, seed)
    if kind == "outputs":
        W = _Walk(_initial_conditions(case["n"], seed))
        W.walk(_beamline(case)[0].elements)
        return dict(label=None, rows=None, margin=W.margin, final=W.S, counts=None, steps=None)
    if kind == "trajectories":
        bl, xd, vd = _beamline(case)
        n = case["n"] // 100 * 100
        W = _Walk(_drawn_ics(n, seed, xd, vd), keep_rows=True)
        W.walk(bl.elements)
        pos = np.full(n, -1)
        pos[W.alive] = np.arange(W.alive.size)
        rows = [[] for _ in W.alive]
        for i, S in W.trace[0]:
            sel = np.flatnonzero(pos[i] >= 0)
            for c in sel:
                rows[pos[i[c]]].append(S[:, c])
        out = np.full((case["n"] // 10_000 + 32, 640, 10), np.nan)
        for k, r in enumerate(rows):
            out[k, :len(r)] = r
        return dict(counts=None, rows=out)
    return None  # counts alone are whole numbers; a drawn gradient's molecules are too many for plain numpy
