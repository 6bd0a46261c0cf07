"""Performance cases of the tracker: what users have it do, through its public
entry points, over the range of sizes, precisions and pushers they meet.

Beams and maps are those of the benchmark's configurations, generated on the
GPU from the seed:

* ``quad``       ~1 MeV protons in a quadrupole-solenoid B map (+-5 cm);
* ``rf_gap``     1 MeV protons crossing a 20 cm RF gap (Ez, Bz), 100 MHz;
* ``electrons``  10 keV-10 MeV electrons in a radial E + solenoid B map (+-10 cm);
* ``ring``       5 MeV protons circulating in a four-sector Bz map (1 m cube).

Kinds of case: ``push`` (``Pusher.push_batch``: one step at a time from a
user's own loop), ``single`` (``Pusher.track``: one particle), ``track``
(``Pusher.track_batch``, also with an electrode assembly) and ``charge``
(``SpaceChargeSolver.solve_device``: deposit, Poisson solve, field).
"""
import math
from types import SimpleNamespace

import numpy as np
import torch

from pypatools_b200 import ElectrodeSurface, Field, Pusher, RFModulation
from pypatools_b200.space_charge import PoissonSolverConfig, SpaceChargeSolver

C = 299792458.0
EPS0 = 8.8541878188e-12
PROTON = dict(q_over_m=9.5788331430e7, mass_mev=938.27208943)
ELECTRON = dict(q_over_m=-1.75882000838e11, mass_mev=0.51099895069)

# beam -> particle, half size of the map's cube [m], time step [s], RF
BEAMS = {
    "quad": dict(ion=PROTON, half=0.05, dt=1e-11, rf=None),
    "rf_gap": dict(ion=PROTON, half=0.1, dt=1e-11, rf=1e8),
    "electrons": dict(ion=ELECTRON, half=0.1, dt=1e-12, rf=None),
    "ring": dict(ion=PROTON, half=0.5, dt=1e-10, rf=None),
}


def listed():
    return [
        # one step of a small bunch: a user's own stepping loop, numpy in and out
        dict(name="push_1000", kind="push", beam="quad", nodes=65, algorithm="boris", precision="fp64", n=1000),
        # a reference trajectory: one proton, every step kept
        dict(name="one_proton", kind="single", beam="quad", nodes=65, algorithm="boris", precision="fp64",
             nsteps=1000, rec=1),
        # the small-bunch configuration: 4096 protons, numpy histories
        dict(name="bunch_4096", kind="track", beam="quad", nodes=65, algorithm="boris", precision="fp64", n=4096,
             nsteps=1000, rec=10, snapshot="host", surface=False),
        # the RF-gap configuration in the default (float64) form with numpy histories
        dict(name="rf_gap_fp64", kind="track", beam="rf_gap", nodes=256, algorithm="boris", precision="fp64",
             n=1000003, nsteps=2000, rec=500, snapshot="host", surface=False),
        # the headline configuration: mixed precision, a large bunch, histories left on the GPU
        dict(name="rf_gap_mixed", kind="track", beam="rf_gap", nodes=256, algorithm="boris", precision="mixed",
             n=6000000, nsteps=2000, rec=500, snapshot="device", surface=False),
        # the electron configuration with the reference's relativistic pushers and the published Vay
        dict(name="electrons_rk4_rel", kind="track", beam="electrons", nodes=129, algorithm="rk4_rel",
             precision="fp64", n=1000000, nsteps=200, rec=200, snapshot="device", surface=False),
        dict(name="electrons_vay_rel", kind="track", beam="electrons", nodes=129, algorithm="vay_rel",
             precision="fp64", n=400001, nsteps=500, rec=100, snapshot="device", surface=False),
        dict(name="electrons_vay_mixed", kind="track", beam="electrons", nodes=129, algorithm="vay",
             precision="mixed", n=1000000, nsteps=1000, rec=1000, snapshot="device", surface=False),
        # the circulating-beam configuration: a map larger than L2, never field-free
        dict(name="ring_mixed", kind="track", beam="ring", nodes=512, algorithm="boris", precision="mixed",
             n=5000000, nsteps=1000, rec=1000, snapshot="device", surface=False),
        # losses on an aperture plate and a beam pipe
        dict(name="electrodes", kind="track", beam="quad", nodes=65, algorithm="boris", precision="fp64",
             n=1000000, nsteps=1000, rec=1000, snapshot="device", surface=True),
        # the space-charge step of a bunch, in free space and inside conductors
        dict(name="charge_open", kind="charge", nx=64, ny=64, nz=128, n=2000000, tol=1e-6, conductors=False),
        dict(name="charge_pipe", kind="charge", nx=64, ny=64, nz=128, n=1000000, tol=1e-6, conductors=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# relative cost of a particle-step, to keep drawn cases below the largest listed one
_WEIGHT = {"boris": 1, "boris_rel": 1.5, "vay": 5, "vay_rel": 4, "rk4": 5, "rk4_rel": 15}


def draw(rng):
    kind = rng.choice(["push", "single", "track", "track", "track", "track", "charge"])
    if kind == "charge":
        pipe = rng.random() < 0.5
        top = 64 if pipe else 96
        return dict(kind="charge", nx=rng.randint(17, top), ny=rng.randint(17, top), nz=rng.randint(24, 128),
                    n=_log_int(rng, 1e4, 4e6), tol=rng.choice([1e-6, 1e-6, 1e-8]), conductors=pipe)
    beam = rng.choice(["quad", "rf_gap", "electrons", "ring"])
    nodes = {"quad": rng.randint(33, 97), "rf_gap": rng.randint(64, 256), "electrons": rng.randint(65, 129),
             "ring": rng.randint(128, 512)}[beam]
    precision = rng.choice(["fp64", "fp64", "mixed"])
    algorithm = rng.choice(["boris", "boris", "boris_rel", "vay", "rk4", "rk4_rel"])
    if precision == "fp64" and rng.random() < 0.25:
        algorithm = "vay_rel"
    if kind == "push":
        return dict(kind=kind, beam=beam, nodes=nodes, algorithm=algorithm, precision=precision,
                    n=_log_int(rng, 1, 30000))
    if kind == "single":
        return dict(kind=kind, beam=beam, nodes=nodes, algorithm=algorithm, precision=precision,
                    nsteps=_log_int(rng, 100, 4000), rec=rng.choice([1, 1, 7, 50]))
    surface = beam == "quad" and algorithm == "boris" and rng.random() < 0.7
    nsteps = _log_int(rng, 100, 2000)
    most = 4e9 / _WEIGHT[algorithm] / nsteps / (10 if surface else 1)
    n = _log_int(rng, 500, max(1000, min(2e6, most)))
    rec = rng.choice([nsteps, max(1, nsteps // 4), max(1, nsteps // rng.randint(5, 9))])
    return dict(kind="track", beam=beam, nodes=nodes, algorithm=algorithm, precision=precision, n=n, nsteps=nsteps,
                rec=rec, snapshot=rng.choice(["host", "device"]), surface=surface)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _speed(ke_mev, mass_mev):
    g = 1.0 + ke_mev / mass_mev
    return C * torch.sqrt(1.0 - 1.0 / (g * g))


def _bunch(case, seed):
    """(r0, v0, phase) of the case's beam: (n, 3), (n, 3) and (n,) float64 on the GPU."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = case.get("n", 1)
    mass = BEAMS[case["beam"]]["ion"]["mass_mev"]

    def normal(s, k=1):
        return s * torch.randn((n, k), generator=gen, device="cuda", dtype=torch.float64)

    def uniform(a, b, k=1):
        return a + (b - a) * torch.rand((n, k), generator=gen, device="cuda", dtype=torch.float64)

    one = torch.ones((n, 1), device="cuda", dtype=torch.float64)
    phase = None
    if case["beam"] == "quad":
        ke = uniform(0.9, 1.1)
        d = torch.cat([normal(5e-3, 2), one], 1)
        r = uniform(-0.01, 0.01, 3)
    elif case["beam"] == "rf_gap":
        ke = uniform(0.99, 1.01)
        d = torch.cat([normal(2e-3, 2), one], 1)
        span = 0.5 * float(_speed(torch.tensor(1.0), mass)) / 1e8
        r = torch.cat([normal(1e-3, 2), uniform(-span, span)], 1)
        phase = uniform(0.0, 2.0 * math.pi)[:, 0].contiguous()
    elif case["beam"] == "electrons":
        ke = 10.0 ** uniform(-2.0, 1.0)
        d = normal(1.0, 3)
        r = normal(2e-3, 3)
    else:
        ke = 5.0 * uniform(0.995, 1.005)
        d = torch.cat([normal(3e-3), -one, normal(3e-3)], 1)
        p = math.sqrt(25.0 + 10.0 * mass) * 1e6 / C                    # B rho of 5 MeV [T m]
        r_eq = (1.0 - math.sqrt(1.0 - 0.2 * p)) / 0.1                  # r (1 - 0.05 r) = B rho
        r = normal(3e-3, 3) + torch.tensor([r_eq, 0.0, 0.0], device="cuda", dtype=torch.float64)
    v = d / d.norm(dim=1, keepdim=True) * _speed(ke, mass)
    return r.contiguous(), v.contiguous(), phase


def _map(case, seed):
    """Node coordinates of one axis and the E and B node values {component: (nodes,)*3 tensor}
    (float64 for the small maps, float32 for the large ones); the seed sets the strength."""
    m = case["nodes"]
    half = BEAMS[case["beam"]]["half"]
    s = 1.0 + 0.01 * math.sin(seed)
    dt = torch.float32 if case["beam"] in ("rf_gap", "ring") else torch.float64
    axis = np.linspace(-half, half, m)
    g = torch.from_numpy(axis).cuda()
    x, y, z = g[:, None, None], g[None, :, None], g[None, None, :]

    def full(a):
        return (s * a).to(dt).expand(m, m, m).contiguous()

    one = torch.ones((1, 1, 1), device="cuda", dtype=torch.float64)
    if case["beam"] == "quad":
        return axis, None, {"x": full(10.0 * y), "y": full(10.0 * x), "z": full(one)}
    if case["beam"] == "rf_gap":
        return axis, {"z": full(5e6 * torch.sin(math.pi * (z + half) / (2 * half)))}, {"z": full(0.2 * one)}
    if case["beam"] == "electrons":
        return axis, {"x": full(1e7 * x), "y": full(1e7 * y)}, {"z": full(0.5 * torch.cos(math.pi * z / (2 * half)))}
    b = 1.0 + 0.1 * torch.cos(4.0 * torch.atan2(y, x)) - 0.05 * torch.sqrt(x * x + y * y)
    return axis, None, {"z": full(b)}


def _charge_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = case["n"]
    p = torch.randn((n, 3), generator=gen, device="cuda", dtype=torch.float64) * 1e-3
    p[:, 2] = 0.14 * (torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) - 0.5)
    q = 1.602176634e-15 * (0.5 + torch.rand(n, generator=gen, device="cuda", dtype=torch.float64))
    return p, q


EXTENT = (0.02, 0.02, 0.3)


def prepare(case, seed):
    if case["kind"] == "charge":
        p, q = _charge_inputs(case, seed)
        assembly = None
        if case["conductors"]:
            # a beam pipe (wall 8-9.5 mm) and a 2 mm thick aperture plate (3 mm hole)
            assembly = ElectrodeSurface.annular_cylinder(0.008, 0.0095, -0.15, 0.15, n_phi=64, n_z=60) + \
                ElectrodeSurface.annular_cylinder(0.003, 0.008, 0.049, 0.051, n_phi=64, n_z=1, n_r=4)
        config = PoissonSolverConfig(EXTENT, (case["nx"], case["ny"], case["nz"]), solver_tol=case["tol"])
        return dict(kind="charge", solver=SpaceChargeSolver(config, electrode_assembly=assembly), p=p, q=q)
    beam = BEAMS[case["beam"]]
    axis, e, b = _map(case, seed)
    grid = {"x": axis, "y": axis, "z": axis}
    r, v, phase = _bunch(case, seed)
    surface = None
    if case.get("surface"):
        surface = ElectrodeSurface.aperture_plate(0.03, 0.005, 0.02, n_phi=48, n_r=3) + \
            ElectrodeSurface.tube(0.012, -0.05, 0.06, n_phi=48, n_z=22)
    ion = SimpleNamespace(name=case["beam"], q_over_m=beam["ion"]["q_over_m"])
    state = dict(kind=case["kind"], dt=beam["dt"], nsteps=case.get("nsteps", 1), rec=case.get("rec", 1),
                 pusher=Pusher(ion, case["algorithm"], electrode_assembly=surface, precision=case["precision"],
                               snapshot=case.get("snapshot", "host")),
                 e=None if e is None else Field.from_arrays(grid, e), b=Field.from_arrays(grid, b),
                 r=r.cpu().numpy(), v=v.cpu().numpy(), rf=None)
    if case["kind"] == "track" and phase is not None:
        state["rf"] = RFModulation(beam["rf"], phase.cpu().numpy())
    return state


def run(s):
    if s["kind"] == "charge":
        return s["solver"].solve_device(s["p"], s["q"])
    if s["kind"] == "push":
        return s["pusher"].push_batch(s["r"], s["v"], s["e"], s["b"], s["dt"])
    if s["kind"] == "single":
        return s["pusher"].track(s["r"][0], s["v"][0], s["e"], s["b"], s["nsteps"], s["dt"], s["rec"])
    return s["pusher"].track_batch(s["r"], s["v"], s["e"], s["b"], s["nsteps"], s["dt"], s["rec"], rf=s["rf"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
# floating-point operations of one update (interpolation apart), FMA = 2
_FLOPS = {"boris": 60, "boris_rel": 80, "vay": 110, "vay_rel": 120, "rk4": 130, "rk4_rel": 230}
_COMPONENTS = {"quad": 3, "rf_gap": 2, "electrons": 3, "ring": 1}


def work(case):
    if case["kind"] == "charge":
        m = case["nx"] * case["ny"] * case["nz"]
        # particles in, potential and field out, and the nodes of one deposit; per unknown about
        # what one multigrid solve to the tolerance costs
        return {"bytes": 32.0 * case["n"] + 40.0 * m, "flops": 60.0 * case["n"] + 1000.0 * m}
    n, k = case.get("n", 1), case.get("nsteps", 1)
    comps = _COMPONENTS[case["beam"]]
    evals = 4 if case["algorithm"].startswith("rk4") else 1
    # the share of the steps inside the map: the gap is crossed in about 1000 steps
    inside = min(1.0, 1000.0 / k) if case["beam"] == "rf_gap" else 1.0
    flops = n * k * inside * (_FLOPS[case["algorithm"]] + evals * (9 + 14 * comps))
    rows = (k // case.get("rec", 1) + 1) if case["kind"] != "push" else 1
    size = 8 if case["precision"] == "fp64" else 4
    touched = min(case["nodes"] ** 3, 8 * n * k) * comps * size
    return {"bytes": 48.0 * n * (1 + rows) + touched, "flops": flops}


# ---------------------------------------------------------------------------
# the same in plain torch, float64
# ---------------------------------------------------------------------------
class _Fields:
    """E and B of the case at points: trilinear, zero outside the map."""

    def __init__(self, case, seed, phase):
        self.axis, e, b = _map(case, seed)
        self.lo, self.hi, self.m = float(self.axis[0]), float(self.axis[-1]), case["nodes"]
        self.g = torch.from_numpy(self.axis).cuda()
        self.names = [("e", c) for c in (e or {})] + [("b", c) for c in b]
        self.values = [(e if k == "e" else b)[c].reshape(-1).double() for k, c in self.names]
        self.omega = 2.0 * math.pi * (BEAMS[case["beam"]]["rf"] or 0.0)
        self.phase = phase

    def __call__(self, r, t):
        inside = ((r >= self.lo) & (r <= self.hi)).all(dim=1)
        d = (self.hi - self.lo) / (self.m - 1)
        cell = torch.floor((r.clamp(self.lo, self.hi) - self.lo) / d).long().clamp(0, self.m - 2)
        w = ((r - self.g[cell]) / (self.g[cell + 1] - self.g[cell])).clamp(0.0, 1.0)
        base = (cell[:, 0] * self.m + cell[:, 1]) * self.m + cell[:, 2]
        u = 1.0 - w
        out = {"e": torch.zeros_like(r), "b": torch.zeros_like(r)}
        for (kind, c), val in zip(self.names, self.values):
            def at(i, j, k):
                return val[base + (i * self.m + j) * self.m + k]
            low = [[at(0, j, k) * u[:, 0] + at(1, j, k) * w[:, 0] for k in (0, 1)] for j in (0, 1)]
            mid = [low[0][k] * u[:, 1] + low[1][k] * w[:, 1] for k in (0, 1)]
            f = mid[0] * u[:, 2] + mid[1] * w[:, 2]
            out[kind][:, "xyz".index(c)] = torch.where(inside, f, 0.0)
        if self.phase is not None:
            out["e"] = out["e"] * torch.cos(self.omega * t + self.phase)[:, None]
        return out["e"], out["b"]


def _dot(a, b):
    return (a * b).sum(dim=1, keepdim=True)


def _gamma_u(u):
    return torch.sqrt(1.0 + _dot(u, u) / (C * C))


def _gamma_v(v):
    return 1.0 / torch.sqrt(1.0 - (_dot(v, v) / (C * C)).clamp(max=0.9999))


def _limit(v):
    s = torch.sqrt(_dot(v, v))
    return torch.where(s >= 0.9999 * C, v * (0.9999 * C / s), v)


def _cross(a, b):
    return torch.linalg.cross(a, b)


def _rotate(w, t):
    wp = w + _cross(w, t)
    return w + _cross(wp, t * (2.0 / (1.0 + _dot(t, t))))


def _kick(alg, w, e, b, dt, qm):
    """The velocity (boris, vay_rel) or u = gamma v (boris_rel, vay) update."""
    if alg == "boris":
        k = 0.5 * qm * dt * e
        return _rotate(w + k, 0.5 * qm * dt * b) + k
    if alg == "boris_rel":
        k = 0.5 * qm * dt * e
        um = w + k
        return _rotate(um, (0.5 * qm * dt) * b / _gamma_u(um)) + k
    if alg == "vay":
        up = w + qm * dt * (e + 0.5 * _cross(w / _gamma_u(w), b))
        tau = 0.5 * qm * dt * b
        tau2, us = _dot(tau, tau), _dot(up, tau) / C
        sigma = 1.0 + _dot(up, up) / (C * C) - tau2
        t = tau / torch.sqrt(0.5 * (sigma + torch.sqrt(sigma * sigma + 4.0 * (tau2 + us * us))))
        return (up + _dot(up, t) * t + _cross(up, t)) / (1.0 + _dot(t, t))
    u = _gamma_v(w) * w                                                # vay_rel, as the reference writes it
    tau = 0.5 * qm * dt * b
    up = u + qm * dt * e
    gis = (1.0 - _dot(up, up) / (C * C)).clamp(min=1e-10)
    tau2, us = _dot(tau, tau), _dot(up, tau) / C
    sigma = gis - tau2
    gn = torch.sqrt(0.5 * (sigma + torch.sqrt(sigma * sigma + 4.0 * (tau2 + us * us))))
    t = tau / gn
    s = t * (2.0 / (1.0 + tau2 / (gn * gn)))
    return _limit((up + _cross(up + _cross(up, t), s)) / gn)


def _slope(alg, v, e, b, qm):
    f = qm * (e + _cross(v, b))
    if alg == "rk4":
        return f
    g = _gamma_v(v)
    return f / g - (_dot(v, f) / (g * C * C)) * v


def _step(alg, r, w, fields, t, dt, qm):
    if alg.startswith("rk4"):
        k1 = _slope(alg, w, *fields(r, t), qm)
        v2 = w + 0.5 * dt * k1
        k2 = _slope(alg, v2, *fields(r + 0.5 * dt * w, t + 0.5 * dt), qm)
        v3 = w + 0.5 * dt * k2
        k3 = _slope(alg, v3, *fields(r + 0.5 * dt * v2, t + 0.5 * dt), qm)
        v4 = w + dt * k3
        k4 = _slope(alg, v4, *fields(r + dt * v3, t + dt), qm)
        r = r + dt / 6.0 * (w + 2.0 * v2 + 2.0 * v3 + v4)
        w = w + dt / 6.0 * (k1 + 2.0 * k2 + 2.0 * k3 + k4)
        return r, (_limit(w) if alg == "rk4_rel" else w)
    w = _kick(alg, w, *fields(r, t), dt, qm)
    return r + dt * (w / _gamma_u(w) if alg in ("boris_rel", "vay") else w), w


def _track(case, seed):
    r, v, phase = _bunch(case, seed)
    beam = BEAMS[case["beam"]]
    alg, dt, qm = case["algorithm"], beam["dt"], beam["ion"]["q_over_m"]
    push = case["kind"] == "push"
    fields = _Fields(case, seed, phase if case["kind"] == "track" else None)
    nsteps, rec = case.get("nsteps", 1), case.get("rec", 1)
    proper = alg in ("boris_rel", "vay")
    w = v / torch.sqrt((1.0 - torch.sqrt(_dot(v, v)) / C) * (1.0 + torch.sqrt(_dot(v, v)) / C)) if proper else v

    def velocity():
        return w / _gamma_u(w) if proper else w

    staggered = alg in ("boris", "boris_rel", "vay") and not push
    if staggered:
        w = _kick(alg, w, *fields(r, 0.0), -0.5 * dt, qm)
    rows_r, rows_v = [r], [velocity()]
    for k in range(nsteps):
        r, w = _step(alg, r, w, fields, k * dt, dt, qm)
        if (k + 1) % rec == 0:
            rows_r.append(r)
            rows_v.append(velocity())
    if push:
        return r, velocity()
    if staggered:
        w = _kick(alg, w, *fields(r, nsteps * dt), 0.5 * dt, qm)
        rows_v[-1] = velocity()
    return torch.stack(rows_r), torch.stack(rows_v)


def _sines(n, h):
    """Eigenvectors and eigenvalues of the zero-boundary second difference on n cells."""
    k = torch.arange(1, n + 1, device="cuda", dtype=torch.float64)
    s = torch.sin(math.pi * torch.remainder(k[:, None] * k[None, :], 2 * (n + 1)) / (n + 1))
    return s * math.sqrt(2.0 / (n + 1)), (2.0 - 2.0 * torch.cos(math.pi * k / (n + 1))) / (h * h)


def _charge(case, seed):
    p, q = _charge_inputs(case, seed)
    cells = [case["nx"], case["ny"], case["nz"]]
    h = [ext / c for ext, c in zip(EXTENT, cells)]
    rho = torch.zeros(cells[0] * cells[1] * cells[2], device="cuda", dtype=torch.float64)
    at, frac = [], []
    for a in range(3):
        x = ((p[:, a] + EXTENT[a] / 2) / h[a]).clamp(0.0, cells[a] - 1.0)
        i = torch.floor(x)
        frac.append(x - i)
        at.append(i.clamp(0, cells[a] - 2).long())
    for i in (0, 1):
        for j in (0, 1):
            for k in (0, 1):
                share = q
                for a, up in enumerate((i, j, k)):
                    share = share * (frac[a] if up else 1.0 - frac[a])
                rho.index_add_(0, ((at[0] + i) * cells[1] + at[1] + j) * cells[2] + at[2] + k, share)
    f = (rho / (h[0] * h[1] * h[2]) / EPS0).reshape(cells)
    (sx, lx), (sy, ly), (sz, lz) = (_sines(c, d) for c, d in zip(cells, h))

    def transform(a):      # the sine matrices are symmetric and their own inverses
        a = torch.tensordot(sx, a, dims=1)
        return torch.matmul(sy, a) @ sz

    phi = transform(transform(f) / (lx[:, None, None] + ly[None, :, None] + lz[None, None, :]))
    e = torch.zeros((3, *cells), device="cuda", dtype=torch.float64)
    inner = (slice(1, -1),) * 3
    for a in range(3):
        n = cells[a]
        diff = (phi.narrow(a, 2, n - 2) - phi.narrow(a, 0, n - 2)) / (2 * h[a])
        cut = tuple(slice(None) if d == a else slice(1, -1) for d in range(3))
        e[(a,) + inner] = -diff[cut]
    return phi, e


def exact(case, seed):
    if case["kind"] == "charge":
        return None if case["conductors"] else _charge(case, seed)
    if case.get("surface"):
        return None
    r, v = _track(case, seed)
    if case["kind"] == "single":
        return r[:, 0].cpu().numpy(), v[:, 0].cpu().numpy()
    if case["kind"] == "push":
        return r.cpu().numpy(), v.cpu().numpy()
    if case["snapshot"] == "host":
        return r.cpu().numpy(), v.cpu().numpy(), None
    return r, v, None
