"""What is timed: time steps of the SD-MHD path through its public entry points.

A case is one of four kinds of call that a user of the framework makes:

* ``steps``  -- ``Solver.step_host(Qin, Qout, nsteps)``: a state from pinned host memory, a
  number of time steps (RK stages, CT projection, norms on the first of ten), the state back
  in pinned host memory.  With one step it is the drop-in for a host code that keeps its
  state in host memory; with ten the copies are a small part and the resident steps count.
* ``resid``  -- ``upload`` + ``compresid`` + the residual array: the drop-in residual
  evaluation of a host code that does its own time stepping.
* ``batch``  -- ``Batch``: a mixed ensemble (orders, sizes, problems) advanced together, every
  solve's state uploaded before and downloaded after.

The states are seeded perturbations of the problems' initial data (density, pressure,
velocity and A_z), with steep fronts where a case asks for them (the artificial viscosity is
on in their cells, as in a run past its first shocks).  The mesh and the bound solver are
what a user's program keeps.
"""
import math
import os
import random
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if os.path.join(ROOT, "chorus-mhd_gb300") not in sys.path:
    sys.path.insert(0, os.path.join(ROOT, "chorus-mhd_gb300"))

from chorus_mhd import Batch, Mesh, Solver, meshgen  # noqa: E402


def _steps(name, problem, nx, ny, N, nsteps, jitter=0.0, k_stage=3, mu=0.0, eta0=0.0, artiv=1, fronts=0, kind="steps"):
    return dict(name=name, kind=kind, problem=problem, nx=nx, ny=ny, N=N, nsteps=nsteps, jitter=jitter, k_stage=k_stage,
                mu=mu, eta0=eta0, artiv=artiv, fronts=fronts)


def listed():
    return [
        # the smallest call: one residual evaluation for a host code, a latency measurement
        _steps("residual 20x18 N4", "orszag_tang", 20, 18, 4, 1, jitter=0.1, kind="resid"),
        # one small solve of an ensemble or of a convergence study, resident for ten steps
        _steps("alfven 32x32 N3", "alfven", 32, 32, 3, 10),
        # the 64x64 Orszag-Tang vortex after its shocks have formed: viscosity on in part of the cells
        _steps("orszag-tang 64x64 N4 fronts", "orszag_tang", 64, 64, 4, 10, fronts=3),
        # an odd mesh at high order
        _steps("orszag-tang 75x53 N6", "orszag_tang", 75, 53, 6, 10, jitter=0.1),
        # physical viscosity and resistivity: every cell carries the gradient and viscous passes
        _steps("viscous 128x128 N5", "orszag_tang", 128, 128, 5, 10, jitter=0.1, mu=1e-3, eta0=1e-3),
        # the MHD rotor on a FREE boundary, gamma 1.4, viscosity on around the disc
        _steps("rotor 256x256 N4", "rotor", 256, 256, 4, 10, jitter=0.1),
        # low order, the other Runge-Kutta scheme, odd sizes
        _steps("five-stage 301x277 N3", "orszag_tang", 301, 277, 3, 10, jitter=0.1, k_stage=5, fronts=2),
        # the highest order
        _steps("orszag-tang 101x90 N8", "orszag_tang", 101, 90, 8, 10, jitter=0.05),
        # the large single solve the benchmark is quoted on, resident
        _steps("orszag-tang 512x512 N5", "orszag_tang", 512, 512, 5, 10, jitter=0.15),
        # the same kind of solve with its state in host memory: copies every step
        _steps("host state 400x400 N5", "orszag_tang", 400, 400, 5, 1, jitter=0.15),
        # a mixed ensemble advanced together
        dict(name="ensemble of 16", kind="batch", count=16, lo=24, hi=96, mix=2024, nsteps=10),
    ]


def draw(rng):
    kind = rng.choice(["steps"] * 6 + ["resid", "batch"])
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(3, 16), lo=rng.randint(8, 24), hi=rng.randint(32, 96),
                    mix=rng.randrange(1 << 20), nsteps=rng.randint(1, 10))
    problem = rng.choice(["orszag_tang", "orszag_tang", "rotor", "alfven"])
    N = rng.choice([2, 3, 4, 4, 5, 5, 6, 7, 8])
    lo = max(8, math.ceil(192 / N)) if problem == "rotor" else 6
    cap = 1.2e6 / (N * N)  # cells of the largest drawn mesh
    side = math.exp(rng.uniform(math.log(lo), math.log(max(lo + 1.0, math.sqrt(cap)))))
    ratio = 1.0 if problem == "rotor" else math.exp(rng.uniform(-0.4, 0.4))
    nx, ny = max(4, round(side * ratio)), max(4, round(side / ratio))
    visc = rng.random() < 0.2
    return dict(kind=kind, problem=problem, nx=nx, ny=ny, N=N, nsteps=1 if kind == "resid" else rng.choice([1, 3, 10]),
                jitter=0.0 if problem == "alfven" else rng.choice([0.0, 0.1, 0.15]), k_stage=rng.choice([3, 3, 5]),
                mu=1e-3 if visc else 0.0, eta0=1e-3 if visc else 0.0, artiv=rng.choice([1, 1, 1, 0]),
                fronts=rng.choice([0, 0, 2]) if problem == "orszag_tang" else 0)


def _members(case):
    """The solves of a batch case, as `steps` cases (16 to 96 cells a side, N = 3..6)."""
    r = random.Random(case["mix"])
    out = []
    for _ in range(case["count"]):
        N = r.randint(3, 6)
        problem = r.choice(["orszag_tang", "rotor", "alfven"])
        side = round(math.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]))))
        if problem == "rotor":
            side = max(side, math.ceil(192 / N))
        out.append(_steps("", problem, side, side, N, case["nsteps"], jitter=0.0 if problem == "alfven" else 0.1))
    return out


# ---------------------------------------------------------------------------
# inputs: mesh vertices, solution points, states (plain numpy and torch)
# ---------------------------------------------------------------------------
SHARED_ANGLE = math.radians(30.0)
LENGTHS = {"orszag_tang": (2 * math.pi, 2 * math.pi), "rotor": (1.0, 1.0),
           "alfven": (1.0 / math.cos(SHARED_ANGLE), 1.0 / math.sin(SHARED_ANGLE))}
GAMMA = {"orszag_tang": 5.0 / 3, "rotor": 1.4, "alfven": 5.0 / 3}
B0 = {"orszag_tang": (0.0, 0.0), "rotor": (0.0, 0.0), "alfven": (math.cos(SHARED_ANGLE), math.sin(SHARED_ANGLE))}
MESH_SEED = 1


def _digits12(a):
    """The values as the vertex file spells them (12 significant digits)."""
    return np.array([float("%.11E" % v) for v in a.ravel()]).reshape(a.shape)


def _vertices(case):
    nx, ny = case["nx"], case["ny"]
    lx, ly = LENGTHS[case["problem"]]
    X, Y = np.meshgrid(np.arange(nx + 1) * (lx / nx), np.arange(ny + 1) * (ly / ny), indexing="xy")
    X[:, -1], Y[-1, :] = lx, ly
    if case["jitter"] > 0:
        rng = np.random.default_rng(MESH_SEED)
        dx = rng.uniform(-case["jitter"], case["jitter"], size=X.shape) * (lx / nx)
        dy = rng.uniform(-case["jitter"], case["jitter"], size=Y.shape) * (ly / ny)
        X[1:-1, 1:-1] += dx[1:-1, 1:-1]
        Y[1:-1, 1:-1] += dy[1:-1, 1:-1]
    return _digits12(X), _digits12(Y)


def _dt(case):
    """CFL 0.1 on the unjittered cell and a bound of the initial wave speed."""
    lx, ly = LENGTHS[case["problem"]]
    speed = {"orszag_tang": 3.2, "rotor": 4.5, "alfven": 1.5}[case["problem"]]
    h = min(lx / case["nx"], ly / case["ny"])
    dt = 0.1 * h / (case["N"] * speed)
    if case["mu"] > 0:
        dt = min(dt, 0.02 * (h / case["N"]) ** 2 / case["mu"])
    return dt


def _solution_points(N):
    return 0.5 * (1.0 - np.cos((2 * np.arange(1, N + 1) - 1) * math.pi / (2 * N)))


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _corners(case):
    """The four corner coordinates of every cell, counter-clockwise: two (cells, 4) tensors."""
    out = []
    for V in _vertices(case):
        V = torch.from_numpy(V).to(_device())
        out.append(torch.stack([V[:-1, :-1], V[:-1, 1:], V[1:, 1:], V[1:, :-1]], -1).reshape(-1, 4))
    return out


def _shape(xi, eta):
    return torch.stack([(1 - xi) * (1 - eta), xi * (1 - eta), xi * eta, (1 - xi) * eta])


_GEOMETRY = {}


def _points(case):
    """Coordinates (cells, N, N) of the solution points, [cell][eta][xi]; kept for the latest mesh."""
    key = (case["problem"], case["nx"], case["ny"], case["N"], case["jitter"])
    if key not in _GEOMETRY:
        _GEOMETRY.clear()
        s = torch.from_numpy(_solution_points(case["N"])).to(_device())
        eta, xi = torch.meshgrid(s, s, indexing="ij")
        _GEOMETRY[key] = [torch.tensordot(c, _shape(xi, eta), 1) for c in _corners(case)]
    return _GEOMETRY[key]


def _state(case, seed):
    """Q (cells, N, N, 9) of a seeded perturbation of the problem's initial data."""
    x, y = _points(case)
    lx, ly = LENGTHS[case["problem"]]
    rng = random.Random("%d %s" % (seed, case["problem"]))
    one, zero = torch.ones_like(x), torch.zeros_like(x)

    def wave(top=2):
        """A periodic phase k.x + phi with its wave numbers."""
        kx, ky = rng.randint(1, top) * 2 * math.pi / lx, rng.choice([-1, 1]) * rng.randint(1, top) * 2 * math.pi / ly
        return kx * x + ky * y + rng.uniform(0, 2 * math.pi), kx, ky

    gam = GAMMA[case["problem"]]
    if case["problem"] == "rotor":
        dx, dy = x - 0.5, y - 0.5
        r = torch.sqrt(dx * dx + dy * dy).clamp_min(1e-30)
        f = ((0.115 - r) / 0.015).clamp(0.0, 1.0)
        spin = torch.where(r < 0.1, one / 0.1, f / r)
        rho, u, v, w, p = 1.0 + 9.0 * f, -2.0 * dy * spin, 2.0 * dx * spin, zero, one
        bx, by, bz = one * 5.0 / math.sqrt(4 * math.pi), zero, zero
        az = bx * y
    elif case["problem"] == "alfven":
        ca, sa = math.sqrt(3.0) / 2, 0.5
        ph = 2 * math.pi * (x * ca + y * sa)
        s, c = 0.1 * torch.sin(ph), 0.1 * torch.cos(ph)
        rho, u, v, w, p = one, -s * sa, s * ca, c, 0.1 * one
        bx, by, bz, az = ca - s * sa, sa + s * ca, c, c / (2 * math.pi)
    else:
        rho, u, v, w, p = gam * gam * one, -torch.sin(y), torch.sin(x), zero, gam * one
        bx, by, bz, az = -torch.sin(y), torch.sin(2 * x), zero, 0.5 * torch.cos(2 * x) + torch.cos(y)
    rho = rho * (1 + 0.03 * torch.sin(wave()[0]))
    p = p * (1 + 0.03 * torch.sin(wave()[0]))
    u = u + 0.02 * torch.sin(wave()[0])
    v = v + 0.02 * torch.sin(wave()[0])
    ph, kx, ky = wave()
    az = az + 0.01 * torch.cos(ph)
    bx, by = bx - 0.01 * ky * torch.sin(ph), by + 0.01 * kx * torch.sin(ph)
    for _ in range(case["fronts"]):
        ph, kx, ky = wave(1)
        width = 0.6 * max(lx / case["nx"], ly / case["ny"]) * math.hypot(kx, ky)
        f = torch.tanh(torch.sin(ph) / width)
        rho, p = rho * (1 + 0.15 * f), p * (1 + 0.15 * f)
    e = p / (gam - 1) + 0.5 * rho * (u * u + v * v + w * w) + 0.5 * (bx * bx + by * by + bz * bz)
    return torch.stack([rho, rho * u, rho * v, rho * w, e, bx, by, bz, az], -1)


# ---------------------------------------------------------------------------
# the framework's side
# ---------------------------------------------------------------------------
_MESHES = {}


def _mesh(case):
    """The loaded mesh of a case; that of the latest case (or ensemble) is kept, as a program
    that runs several states on one mesh keeps it."""
    key = tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "kind", "nsteps", "fronts")))
    if key not in _MESHES:
        if len(_MESHES) >= 16:
            _MESHES.clear()
        with tempfile.TemporaryDirectory() as d:
            meshgen.write_case(meshgen.CaseSpec(
                nx=case["nx"], ny=case["ny"], N=case["N"], problem=case["problem"], jitter=case["jitter"], seed=MESH_SEED,
                dt=_dt(case), k_stage=case["k_stage"], mu=case["mu"], eta0=case["eta0"], artiv=case["artiv"]), d)
            _MESHES[key] = Mesh(d)
    return _MESHES[key]


class _Solve:
    """A bound solver, its state in pinned host memory and a pinned buffer for the result."""

    def __init__(self, case, seed):
        self.solver = Solver(_mesh(case), initial_state=False)
        q = _state(case, seed).reshape(-1)
        self.qin = torch.empty(q.numel(), dtype=torch.float64, pin_memory=q.is_cuda)
        self.qin.copy_(q)
        self.qout = torch.empty(q.numel(), dtype=torch.float64, pin_memory=q.is_cuda)


def prepare(case, seed):
    members = _members(case) if case["kind"] == "batch" else [case]
    solves = [_Solve(c, seed + i) for i, c in enumerate(members)]
    state = {"case": case, "solves": solves}
    if case["kind"] == "batch":
        state["batch"] = Batch()
        for s in solves:
            state["batch"].add(s.solver)
    return state


def run(state):
    case, solves = state["case"], state["solves"]
    if case["kind"] == "batch":
        for s in solves:
            s.solver.upload(s.qin.numpy())
        state["batch"].step(case["nsteps"])
        state["batch"].sync()
        for s in solves:
            s.solver.state(s.qout.numpy())
        return [s.qout for s in solves]
    s = solves[0]
    if case["kind"] == "resid":
        s.solver.upload(s.qin.numpy())
        s.solver.compresid()
        return {"resid": s.solver.array("resid", s.solver.nq), "eigv": s.solver.eigvmax()[0]}
    s.solver.iter, s.solver.ctime = 0, 0.0
    d = s.solver.step_host(s.qin.numpy(), s.qout.numpy(), case["nsteps"])[0]
    return {"Q": s.qout, "eigv": d["eigvmax_g"], "resid_norm": d["residglob"]}


def work(case):
    """Bytes that a step cannot do without: per stage and cell the state and the RK register,
    read and written, each face trace once, the geometry; the CT projection; the copies of a host state.  Operations:
    the flux, divergence and update arithmetic of the scheme as it is written."""
    if case["kind"] == "batch":
        parts = [work(c) for c in _members(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    N, cells = case["N"], case["nx"] * case["ny"]
    stages = 1 if case["kind"] == "resid" else 5 * case["nsteps"]
    per_stage = 216 * N * N + 1728 * N + 144
    ct = 0 if case["kind"] == "resid" else case["nsteps"] * (24 * N * N + 64 * N)
    lines = 2 * N * (9 * N * (N + 1) * 2 + 10 * N * (N + 1) * 2)  # interpolation and derivatives along the lines
    points = 2 * N * (N - 1) * 58 + 2 * N * 230 + 9 * N * N * 4 + 4 * N ** 3
    if case["mu"] > 0:
        lines += 2 * N * (16 * N * (N + 1) * 2) * 2
        points += 2 * N * (N + 1) * 150
    return {"bytes": cells * (stages * per_stage + ct + 2 * 72 * N * N), "flops": cells * stages * (lines + points)}


# ---------------------------------------------------------------------------
# the scheme in plain torch, in 64 bits
# ---------------------------------------------------------------------------
def _lagrange(nodes, at):
    """(len(at), len(nodes)) values of the Lagrange basis."""
    out = np.ones((len(at), len(nodes)))
    for i, xi in enumerate(nodes):
        for s, xs in enumerate(nodes):
            if s != i:
                out[:, i] *= (at - xs) / (xi - xs)
    return out


def _derivative(nodes, at):
    """(len(at), len(nodes)) derivatives of the Lagrange basis."""
    out = np.zeros((len(at), len(nodes)))
    for i, xi in enumerate(nodes):
        for k, xk in enumerate(nodes):
            if k == i:
                continue
            t = np.full(len(at), 1.0 / (xi - xk))
            for s, xs in enumerate(nodes):
                if s not in (i, k):
                    t *= (at - xs) / (xi - xs)
            out[:, i] += t
    return out


def _flux_points(N):
    """0, the Legendre-Gauss points of order N - 1, 1; those of order 6 and 7 to the 12 digits
    that the scheme's definition gives."""
    g = np.polynomial.legendre.leggauss(N - 1)[0] if N > 1 else np.zeros(0)
    if N >= 7:
        g = np.round(g, 12)
    return np.concatenate([[0.0], (1.0 + g) / 2, [1.0]])


class _Scheme:
    """Spectral differences for ideal and resistive MHD on a structured nx x ny mesh."""

    def __init__(self, case):
        self.nx, self.ny, self.N = case["nx"], case["ny"], case["N"]
        self.periodic = case["problem"] != "rotor"
        self.gam, (self.b0x, self.b0y) = GAMMA[case["problem"]], B0[case["problem"]]
        self.mu, self.eta0, self.artiv, self.dt, self.k_stage = case["mu"], case["eta0"], case["artiv"], _dt(case), case["k_stage"]
        dev = _device()
        N = self.N
        xs, xf = _solution_points(N), _flux_points(N)
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
        self.xf, self.L, self.D = t(xf), t(_lagrange(xs, xf)), t(_derivative(xf, xs))
        low = _solution_points(N - 1)
        self.A = t(_lagrange(low, xs) @ _lagrange(xs, low))
        cx, cy = _corners(case)

        def metric(xi, eta):
            """Rows of the metric at points (..): (x_xi, y_xi, x_eta, y_eta)."""
            a = torch.stack([eta - 1, 1 - eta, eta, -eta])
            b = torch.stack([xi - 1, -xi, xi, 1 - xi])
            return [torch.tensordot(c, m, 1) for m in (a, b) for c in (cx, cy)]

        grid = lambda e, x: torch.meshgrid(e, x, indexing="ij")  # noqa: E731
        s, f = t(xs), self.xf
        eta, xi = grid(s, s)
        xxi, yxi, xet, yet = metric(xi, eta)
        self.J = xxi * yet - xet * yxi
        eta, xi = grid(s, f)
        _, _, xet, yet = metric(xi, eta)
        self.S1 = torch.stack([yet, -xet], -1)
        eta, xi = grid(f, s)
        xxi, yxi, _, _ = metric(xi, eta)
        self.S2 = torch.stack([-yxi, xxi], -1)
        lx, ly = (float("%.11E" % v) for v in LENGTHS[case["problem"]])
        self.h = math.sqrt(lx * ly / (self.nx * self.ny))

    # -- lines
    def to_flux(self, q):
        """Values at the flux points of the xi lines [cell][eta][f] and of the eta lines [cell][f][xi]."""
        return torch.einsum("fi,cji...->cjf...", self.L, q), torch.einsum("fj,cji...->cfi...", self.L, q)

    def divergence(self, a, b):
        return torch.einsum("if,cjf...->cji...", self.D, a) + torch.einsum("jf,cfi...->cji...", self.D, b)

    # -- faces: (lower cell's trace, upper cell's trace) pairs along xi and eta
    def sides(self, a, b):
        """Traces (ny, nx, N, ...) of every cell: right, left, top, bottom."""
        g = lambda z: z.reshape(self.ny, self.nx, *z.shape[1:])  # noqa: E731
        a, b = g(a), g(b)
        return a[:, :, :, -1], a[:, :, :, 0], b[:, :, -1], b[:, :, 0]

    def faces(self, a, b):
        """Both sides of the two-sided faces: along xi, faces i|i+1 (wrapping if periodic), along eta the same."""
        right, left, top, bottom = self.sides(a, b)
        if self.periodic:
            return (right, torch.roll(left, -1, 1)), (top, torch.roll(bottom, -1, 0))
        return (right[:, :-1], left[:, 1:]), (top[:-1], bottom[1:])

    def set_faces(self, a, b, fx, fy):
        """Put face values on both sides (fx along xi, fy along eta)."""
        a = a.reshape(self.ny, self.nx, *a.shape[1:]).clone()
        b = b.reshape(self.ny, self.nx, *b.shape[1:]).clone()
        if self.periodic:
            a[:, :, :, -1], a[:, :, :, 0] = fx, torch.roll(fx, 1, 1)
            b[:, :, -1], b[:, :, 0] = fy, torch.roll(fy, 1, 0)
        else:
            a[:, :-1, :, -1], a[:, 1:, :, 0] = fx, fx
            b[:-1, :, -1], b[1:, :, 0] = fy, fy
        return a.reshape(-1, *a.shape[2:]), b.reshape(-1, *b.shape[2:])

    def mean_faces(self, a, b):
        (l, r), (d, u) = self.faces(a, b)
        return self.set_faces(a, b, 0.5 * (l + r), 0.5 * (d + u))

    # -- physics
    def flux(self, q, n):
        """Ideal MHD flux along n (..., 2)."""
        rho, m, E, B = q[..., 0], q[..., 1:4], q[..., 4], q[..., 5:8]
        v = m / rho[..., None]
        vn = v[..., 0] * n[..., 0] + v[..., 1] * n[..., 1]
        bn = B[..., 0] * n[..., 0] + B[..., 1] * n[..., 1]
        b2 = (B * B).sum(-1)
        p = (self.gam - 1) * (E - 0.5 * rho * (v * v).sum(-1) - 0.5 * b2)
        pt = p + 0.5 * b2
        fm = m * vn[..., None] - B * bn[..., None]
        fm[..., 0] += pt * n[..., 0]
        fm[..., 1] += pt * n[..., 1]
        fe = (E + pt) * vn - bn * (v * B).sum(-1)
        fb = B * vn[..., None] - v * bn[..., None]
        return torch.cat([(rho * vn)[..., None], fm, fe[..., None], fb], -1), p, vn

    def rusanov(self, ql, qr, S):
        """Flux through faces with area vector S seen from the lower side, the wave speed and the normal velocities."""
        mag = torch.sqrt((S * S).sum(-1))
        n = S / mag[..., None]
        fl, pl, vl = self.flux(ql[..., :8], n)
        fr, pr, vr = self.flux(qr[..., :8], n)
        B = 0.5 * (ql[..., 5:8] + qr[..., 5:8])
        rho = 0.5 * (ql[..., 0] + qr[..., 0])
        ca, cd = self.gam * 0.5 * (pl + pr) / rho, (B * B).sum(-1) / rho
        bn = B[..., 0] * n[..., 0] + B[..., 1] * n[..., 1]
        s = ca + cd
        speed = 0.5 * (vl + vr).abs() + torch.sqrt(0.5 * (s + torch.sqrt(s * s - 4 * ca * bn * bn / rho)))
        return 0.5 * mag[..., None] * (fl + fr - speed[..., None] * (qr - ql)[..., :8]), speed.max(), vl, vr

    def viscous(self, q, g, S, mut):
        """Viscous, resistive and artificial-viscosity flux contracted with S; g (..., 2, 9)."""
        rho, B = q[..., 0], q[..., 5:8]
        v = q[..., 1:4] / rho[..., None]
        dr = g[..., 0]
        dv = (g[..., 1:4] - dr[..., None] * v[..., None, :]) / rho[..., None, None]
        ke = 0.5 * (v * v).sum(-1)
        inner = (q[..., 4] - rho * ke - 0.5 * (B * B).sum(-1)) / rho
        dke = ke[..., None] * dr + rho[..., None] * (v[..., None, :] * dv).sum(-1)
        dpb = (B[..., None, :] * g[..., 5:8]).sum(-1)
        de = (g[..., 4] - dke - dpb - dr * inner[..., None]) / rho[..., None]
        div = dv[..., 0, 0] + dv[..., 1, 1]
        txx = mut * (2 * dv[..., 0, 0] - 2.0 / 3 * div)
        tyy = mut * (2 * dv[..., 1, 1] - 2.0 / 3 * div)
        txy = mut * (dv[..., 0, 1] + dv[..., 1, 0])
        txz, tyz = mut * dv[..., 0, 2], mut * dv[..., 1, 2]
        k = mut * self.gam / 0.72
        jx, jy, jz = g[..., 1, 7], -g[..., 0, 7], g[..., 0, 6] - g[..., 1, 5]
        e = self.eta0
        f = [txx, txy, txz, v[..., 0] * txx + v[..., 1] * txy + v[..., 2] * txz + k * de[..., 0] + e * (jz * B[..., 1] - jy * B[..., 2]),
             0 * jx, e * jz, -e * jy]
        h = [txy, tyy, tyz, v[..., 0] * txy + v[..., 1] * tyy + v[..., 2] * tyz + k * de[..., 1] + e * (jx * B[..., 2] - jz * B[..., 0]),
             -e * jz, 0 * jx, e * jx]
        out = [a * S[..., 0] + b * S[..., 1] for a, b in zip(f, h)]
        return torch.stack([torch.zeros_like(rho)] + out, -1)

    def gradient(self, a, b):
        """(cells, N, N, 2, ...) gradient of face-corrected flux-point values."""
        g = [self.divergence(a * self.S1[..., d, None], b * self.S2[..., d, None]) / self.J[..., None] for d in (0, 1)]
        return torch.stack(g, -2)

    def residual(self, Q):
        a, b = self.to_flux(Q)
        F, _, _ = self.flux(a[..., :8], self.S1)
        G, _, _ = self.flux(b[..., :8], self.S2)
        (l, r), (d, u) = self.faces(a, b)
        (nx, _), (ny, _) = self.faces(self.S1, self.S2)
        fx, e1, vl, _ = self.rusanov(l, r, nx)
        fy, e2, vd, vu = self.rusanov(d, u, ny)
        eig = torch.maximum(e1, e2)
        if not self.periodic:  # FREE faces: the cell's own trace on both sides
            right, left, top, bottom = self.sides(a, b)
            n1, n0, n3, n2 = self.sides(self.S1, self.S2)
            for q, n in ((right[:, -1], n1[:, -1]), (left[:, 0], n0[:, 0]), (top[-1], n3[-1]), (bottom[0], n2[0])):
                eig = torch.maximum(eig, self.rusanov(q, q, n)[1])
        F, G = self.set_faces(F, G, fx, fy)
        # A_z upwinded by the normal velocity of the face's first cell: the lower one, or the
        # bottom row's on the periodic wrap along eta
        zx = torch.where(vl > 0, l[..., 8], r[..., 8])
        zy = torch.where(vd > 0, d[..., 8], u[..., 8])
        if self.periodic:
            zy[-1] = torch.where(vu[-1] < 0, u[-1, ..., 8], d[-1, ..., 8])
        za, zb = self.set_faces(a[..., 8], b[..., 8], zx, zy)
        mut1 = mut2 = None
        if self.artiv:
            rho = Q[..., 0]
            smooth = torch.einsum("jn,im,cnm->cji", self.A, self.A, rho)
            sensor = (((smooth - rho) / rho) ** 2).sum((1, 2))
            eps = eig * self.h / (self.N - 1)
            ramp = 0.5 * eps * (1 + torch.sin(math.pi * (torch.log10(sensor.clamp(1e-6, 0.1)) + 3.5) / 5.0))
            mu = torch.where(sensor < 1e-6, torch.zeros_like(ramp), torch.where(sensor > 0.1, eps, ramp)).reshape(self.ny, self.nx)
            right, left, top, bottom = (mu.clone() for _ in range(4))
            if self.periodic:
                right, left = 0.5 * (mu + torch.roll(mu, -1, 1)), 0.5 * (mu + torch.roll(mu, 1, 1))
                top, bottom = 0.5 * (mu + torch.roll(mu, -1, 0)), 0.5 * (mu + torch.roll(mu, 1, 0))
            else:
                right[:, :-1] = left[:, 1:] = 0.5 * (mu[:, :-1] + mu[:, 1:])
                top[:-1] = bottom[1:] = 0.5 * (mu[:-1] + mu[1:])
            col = lambda z: z.reshape(-1, 1, 1)  # noqa: E731
            mut1 = col(left) * (1 - self.xf) + col(right) * self.xf
            mut2 = col(bottom) * (1 - self.xf[:, None]) + col(top) * self.xf[:, None]
        if self.mu > 0 or self.eta0 > 0 or (self.artiv and bool((mu > 0).any())):
            a, b = self.mean_faces(a, b)
            ga, gb = self.to_flux(self.gradient(a, b))
            ga, gb = self.mean_faces(ga, gb)
            F = F - self.viscous(a, ga, self.S1, self.mu + (mut1 if self.artiv else 0.0))
            G = G - self.viscous(b, gb, self.S2, self.mu + (mut2 if self.artiv else 0.0))
        res = -self.divergence(F, G) / self.J[..., None]
        gz = self.gradient(za[..., None], zb[..., None])[..., 0]
        u, v = Q[..., 1] / Q[..., 0], Q[..., 2] / Q[..., 0]
        adv = -(u * (gz[..., 0] - self.b0y) + v * (gz[..., 1] + self.b0x))
        return torch.cat([res, adv[..., None]], -1), eig

    def project(self, Q):
        """B = B0 + curl A_z from the face-averaged A_z."""
        a, b = self.mean_faces(*self.to_flux(Q[..., 8]))
        g = self.gradient(a[..., None], b[..., None])[..., 0]
        Q = Q.clone()
        Q[..., 5], Q[..., 6] = self.b0x + g[..., 1], self.b0y - g[..., 0]
        return Q

    def step(self, Q):
        """One time step: the state, the last stage's residual norm and wave speed."""
        dt, q0 = self.dt, Q
        if self.k_stage == 5:  # SSPRK(5,4)
            r, _ = self.residual(Q)
            q1 = Q + 0.39175222700392 * dt * r
            r, _ = self.residual(q1)
            q2 = 0.44437049406734 * q0 + 0.55562950593266 * q1 + 0.36841059262959 * dt * r
            r, _ = self.residual(q2)
            q3 = 0.6201018513854 * q0 + 0.3798981486146 * q2 + 0.25189177424738 * dt * r
            r3, _ = self.residual(q3)
            q4 = 0.17807995410773 * q0 + 0.82192004589227 * q3 + 0.54497475021237 * dt * r3
            r, eig = self.residual(q4)
            Q = (0.00683325884039 * q0 + 0.51723167208978 * q2 + 0.12759831133288 * q3 + 0.34833675773694 * q4
                 + 0.08460416338212 * dt * r3 + 0.22600748319395 * dt * r)
        else:  # SSPRK(5,3)
            r, _ = self.residual(Q)
            q1 = Q + 0.377268915331368 * dt * r
            r, _ = self.residual(q1)
            q2 = q1 + 0.377268915331368 * dt * r
            r, _ = self.residual(q2)
            q3 = 0.355909775063327 * q0 + 0.644090224936674 * q2 + 0.242995220537396 * dt * r
            r, _ = self.residual(q3)
            q4 = 0.367933791638137 * q0 + 0.632066208361863 * q3 + 0.238458932846290 * dt * r
            r, eig = self.residual(q4)
            Q = 0.237593836598569 * q2 + 0.762406163401431 * q4 + 0.287632146308408 * dt * r
        return self.project(Q), math.sqrt(float((r * r).sum()) / (Q.shape[0] * self.N * self.N * 5)), float(eig)


def exact(case, seed):
    if case["kind"] == "batch":
        return [exact(c, seed + i)["Q"] for i, c in enumerate(_members(case))]
    if not torch.cuda.is_available() and case["nx"] * case["ny"] * case["N"] ** 2 * case["nsteps"] > 4e6:
        return None
    scheme, Q = _Scheme(case), _state(case, seed)
    if case["kind"] == "resid":
        r, eig = scheme.residual(Q)
        return {"resid": r.reshape(-1), "eigv": float(eig)}
    for k in range(case["nsteps"]):
        Q, norm, eig = scheme.step(Q)
        if k == 0:
            first = norm, eig
    return {"Q": Q.reshape(-1), "eigv": first[1], "resid_norm": first[0]}
