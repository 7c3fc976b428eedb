"""The workloads the solver is timed on, each through its public entry points.

``listed()`` gives the cases, ``draw(rng)`` one more of the same ranges,
``prepare`` what a program holds before the call (a ``Solver`` with its state
on the device, host arrays), ``run`` one pass, ``work`` the bytes and
operations a pass cannot do without and ``exact`` the same outputs in float64
from plain torch.

Kinds of pass:
  step      a stretch of a run: `steps` fused time steps, then what an output
            step reads (fields into pinned host arrays, the radial means when
            statistics run, the conservation sums of a periodic box)
  granular  the same stretch through the five launchers, one by one
  restart   a run continued from host populations: upload, steps, download
  adjoint   gradient of the bubble-shape objective over `steps` steps with
            `snapshots` held states
  jetgrad   gradient of the jet objective with respect to the inlet profile

Flows (densities and velocities come from the seed):
  bubble    one sphere in the middle of the box
  drops     a dozen spheres of different sizes
  jet       a widening, wavy column along y with droplets torn off it, the
            inlet disc at y = 0; inlet perturbation of 1 %
"""
import math

import numpy as np
import torch

from multicomponent_color_gradient_b200 import Solver, derive

Q = 27
CX = [0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 0, 0, 1, -1, 1, -1, 0, 0, 1, -1, 1, -1, 1, -1, -1, 1]
CY = [0, 0, 0, 1, -1, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 1, -1, 1, -1, 1, -1, -1, 1, 1, -1]
CZ = [0, 0, 0, 0, 0, 1, -1, 0, 0, 1, -1, 1, -1, 0, 0, -1, 1, -1, 1, 1, -1, -1, 1, 1, -1, 1, -1]
FIELDS = ("rhor", "rhob", "ux", "uy", "uz")
RADIAL = ("sum_uy", "sum_uy2", "sum_ur", "sum_ur2", "sum_uruy")
U_JET = 0.05
INLET_NOISE = 0.01
LARGEST = 340e6  # node updates of the largest listed case


def listed():
    def c(name, kind, shape, flow, boundary, storage, steps, stats=False, snapshots=0, segment=0):
        return dict(name=name, kind=kind, NX=shape[0], NY=shape[1], NZ=shape[2], flow=flow, boundary=boundary,
                    storage=storage, steps=steps, stats=stats, snapshots=snapshots, segment=segment)

    return [
        # the smallest jet of the test cases: every step is a launch's latency
        c("jet_24x40x24", "step", (24, 40, 24), "jet", "jet", "f32", 20, stats=True),
        # the static bubble of the physics checks, mass and momentum monitored
        c("bubble_64", "step", (64, 64, 64), "bubble", "periodic", "f32", 20),
        # the jet crop used for parameter scans
        c("jet_64x128x64", "step", (64, 128, 64), "jet", "jet", "f32", 20, stats=True),
        # the same jet driven by a host loop over the five launchers
        c("granular_jet_64x128x64", "granular", (64, 128, 64), "jet", "jet", "f32", 10, stats=True),
        # an emulsion in a box with no round size, reduced storage
        c("drops_97x75x131_f16", "step", (97, 75, 131), "drops", "periodic", "f16", 20),
        # a jet whose rows are longer than 128 and not a round number
        c("jet_200x301x183", "step", (200, 301, 183), "jet", "jet", "f32", 10, stats=True),
        # the benchmark's jet
        c("jet_128x256x128", "step", (128, 256, 128), "jet", "jet", "f32", 20, stats=True),
        # the reference's shipped grid with reduced storage
        c("jet_128x400x128_f16", "step", (128, 400, 128), "jet", "jet", "f16", 20, stats=True),
        # the large jet of the production runs
        c("jet_256x512x256", "step", (256, 512, 256), "jet", "jet", "f32", 10, stats=True),
        # a run continued from saved populations
        c("restart_bubble_64", "restart", (64, 64, 64), "bubble", "closed", "f32", 20),
        # one gradient evaluation of the deforming bubble, few held states
        c("adjoint_bubble_96", "adjoint", (96, 96, 96), "bubble", "periodic", "f32", 40, snapshots=8),
        # one gradient evaluation of the inlet profile, in segments
        c("jetgrad_64x128x64", "jetgrad", (64, 128, 64), "jet", "jet", "f32", 40, segment=10),
    ]


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["granular", "restart", "adjoint", "jetgrad"])
    flow, boundary = {
        "adjoint": ("bubble", "periodic"), "jetgrad": ("jet", "jet"), "granular": ("jet", "jet"),
        "restart": ("bubble", "closed"),
    }.get(kind) or rng.choice([("jet", "jet"), ("jet", "jet"), ("drops", "periodic"), ("bubble", "periodic"),
                               ("bubble", "closed")])

    def size(lo, hi):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        return n if rng.random() < 0.5 else max(lo, n // 16 * 16)

    small = kind in ("restart", "adjoint", "jetgrad")
    NX, NZ = size(16, 128 if small else 256), size(16, 128 if small else 256)
    NY = size(16, 128 if small else 512)
    steps = rng.choice([10, 20, 40])
    while steps > 10 and NX * NY * NZ * steps > LARGEST:
        steps //= 2
    while NX * NY * NZ * steps > LARGEST:
        NY = max(16, NY // 2)
    return dict(kind=kind, NX=NX, NY=NY, NZ=NZ, flow=flow, boundary=boundary,
                storage="f32" if kind in ("granular", "restart", "adjoint") else rng.choice(["f32", "f16"]),
                steps=steps, stats=kind == "granular" or (kind == "step" and flow == "jet" and rng.random() < 0.7),
                snapshots=rng.choice([4, 8, steps + 1]) if kind == "adjoint" else 0,
                segment=rng.choice([0, 5, 10]) if kind == "jetgrad" else 0)


# ---------------------------------------------------------------- inputs

def _parameters(case, seed):
    n = min(case["NX"], case["NZ"])
    jet = case["flow"] == "jet"
    return dict(NX=case["NX"], NY=case["NY"], NZ=case["NZ"], boundary=case["boundary"], storage=case["storage"],
                jet_radius=max(2.0, n / 16.0), jet_velocity=U_JET, bubble_radius=n / 4.0,
                tau=0.52 if jet else 0.7, sigma=0.005 if jet else 0.01, beta_recolor=0.8 if jet else 0.7,
                inlet_noise=INLET_NOISE if jet else 0.0, seed=int(seed), NSTATS_START_STEP=10 ** 9,
                NSTEP=10 ** 6, NOUTPUT=1000)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _fields(case, seed):
    """rhor, rhob, ux, uy, uz (float32, [NZ][NY][NX] flattened, ghost shell
    included) of the case's flow."""
    NX, NY, NZ = case["NX"], case["NY"], case["NZ"]
    p = _parameters(case, seed)
    rng = np.random.RandomState(seed % (2 ** 32))
    dev, f = _device(), torch.float32
    x = torch.arange(NX, device=dev, dtype=f).view(1, 1, NX)
    y = torch.arange(NY, device=dev, dtype=f).view(1, NY, 1)
    z = torch.arange(NZ, device=dev, dtype=f).view(NZ, 1, 1)
    L = (NX - 2, NY - 2, NZ - 2)
    axis = (x, y, z)

    def sphere(c, r):
        """Signed distance into the sphere (periodic images when the box is)."""
        d2 = 0.0
        for a, ca, la in zip(axis, c, L):
            d = (a - 1 - ca).abs()
            if case["boundary"] == "periodic":
                d = torch.remainder(d, la)
                d = torch.minimum(d, la - d)
            d2 = d2 + d * d
        return r - d2.sqrt()

    def wave(amplitude):
        """A smooth mode, periodic over the interior."""
        k = rng.randint(-2, 3, 3)
        k[rng.randint(3)] += 1
        phase = float(rng.uniform(0, 2 * np.pi))
        arg = sum(2 * np.pi * float(ki) / la * (a - 1) for ki, la, a in zip(k, L, axis))
        return amplitude * torch.cos(arg + phase)

    if case["flow"] == "jet":
        R = p["jet_radius"]
        dx, dz = x - (NX - 1) / 2.0, z - (NZ - 1) / 2.0
        bend = [float(v) for v in rng.uniform(0, 2 * np.pi, 4)]
        s = y / NY
        cx = 0.4 * R * s * torch.sin(2 * np.pi * 1.5 * s + bend[0])
        cz = 0.4 * R * s * torch.sin(2 * np.pi * 1.5 * s + bend[1])
        r = ((dx - cx) ** 2 + (dz - cz) ** 2).sqrt()
        radius = R * (1 + 0.6 * s + 0.15 * torch.sin(2 * np.pi * 4 * s + bend[2])
                      + 0.1 * torch.sin(2 * np.pi * 9 * s + bend[3]))
        d = radius - r
        for _ in range(8):  # droplets around the downstream half
            a, far = rng.uniform(0, 2 * np.pi), R * rng.uniform(2.2, 3.5)
            c = (L[0] / 2 + far * np.cos(a), L[1] * rng.uniform(0.4, 0.95), L[2] / 2 + far * np.sin(a))
            d = torch.maximum(d, sphere([float(v) for v in c], float(R * rng.uniform(0.25, 0.5))))
    elif case["flow"] == "bubble":
        c = [la / 2.0 + float(rng.uniform(-1, 1)) for la in L]
        d = sphere(c, min(L) / 4.0)
    else:
        d = None
        for _ in range(12):
            s = sphere([float(la * rng.uniform()) for la in L], float(min(L) * rng.uniform(0.08, 0.18)))
            d = s if d is None else torch.maximum(d, s)
    inside = 0.5 * (1.0 + torch.tanh(0.9 * d)) + torch.zeros((NZ, NY, NX), device=dev, dtype=f)
    rhob, rhor = inside, 1.0 - inside
    u = [wave(2e-3) + wave(2e-3) for _ in range(3)]
    if case["flow"] == "jet":
        u = [inside * v for v in u]
        u[1] = u[1] + 0.8 * U_JET * inside
        mask = (((x - (NX - 1) / 2.0) ** 2 + (z - (NZ - 1) / 2.0) ** 2) <= p["jet_radius"] ** 2).to(f)
        rhob[:, 0:1, :] = mask
        rhor[:, 0:1, :] = 1.0 - mask
    elif case["flow"] == "bubble":  # deforming
        u = [a + wave(8e-3) for a in u]
    z0 = torch.zeros((NZ, NY, NX), device=dev, dtype=f)
    return [(v + z0).reshape(-1).cpu().numpy() for v in (rhor, rhob, *u)]


# ---------------------------------------------------------------- a pass

def _pinned(n):
    t = torch.empty(n, dtype=torch.float32)
    if torch.cuda.is_available():
        t = t.pin_memory()
    return t.numpy()


def prepare(case, seed):
    S = Solver(derive(_parameters(case, seed)))
    F = _fields(case, seed)
    S.init_equilibrium(*F)
    state = {"case": case, "solver": S}
    kind = case["kind"]
    if kind in ("step", "granular"):
        if case["stats"]:
            S.set_radial_statistics(1)
        state["out"] = {k: _pinned(S.N) for k in FIELDS}
    elif kind == "restart":
        fr, fb = S.get_populations()
        state["fr"], state["fb"] = _pinned(fr.size), _pinned(fb.size)
        state["fr"][:], state["fb"][:] = fr, fb
        state["fields"] = F
    elif kind == "adjoint":
        state["target"] = (F[0] - F[1]) / (F[0] + F[1])
        state["fields"] = F
    elif kind == "jetgrad":
        S.set_inlet_bessel([0.1, -0.05, 0.02])
    return state


def _radial_means(S):
    R = S.get_radial()
    n = np.maximum(R["count"], 1)
    return {k: (R[k] / n).astype(np.float32) for k in RADIAL}


def run(state):
    case, S, kind = state["case"], state["solver"], state["case"]["kind"]
    if kind == "step":
        S.step(case["steps"])
        out = {"fields": S.get_fields(state["out"])}
        if case["stats"]:
            out["radial"] = _radial_means(S)
        if case["boundary"] == "periodic":
            out["mass"] = S.conservation_sums()[:2].astype(np.float32)
        return out
    if kind == "granular":
        for _ in range(case["steps"]):
            S.launch_Macros()
            S.launch_accumulate_radial_moments()
            S.launch_collistream()
            S.launch_inlet_bc()
            S.launch_neumann_bc()
        return {"fields": S.get_fields(state["out"]), "radial": _radial_means(S)}
    if kind == "restart":
        S.set_fields(*state["fields"])
        S.set_populations(state["fr"], state["fb"])
        S.step(case["steps"])
        fr, fb = S.get_populations()
        return {"fr": fr, "fb": fb, "finite": S.check_finite()}
    if kind == "adjoint":
        S.init_equilibrium(*state["fields"])
        r = S.adjoint_run(state["target"], case["steps"], case["snapshots"])
        return {k: r[k] for k in ("J", "dJ_dsigma", "dJ_dtau", "dJ_du0")}
    t0, y0 = _window(case)
    r = S.adjoint_jet_run(case["steps"], t0, case["steps"] - 1, y0, case["segment"])
    return {"J": r["J"], "dJ_dc": r["dJ_dc"].astype(np.float32)}


def _window(case):
    """First step and first row of the jet objective: rows that the inlet's
    influence (speed of sound) has reached by then."""
    return case["steps"] // 2, max(2, min(case["steps"] // 4, case["NY"] // 2))


def work(case):
    """Populations of both colours read and written once per step (a jet
    gradient's reverse step: lambda read and written, the moment record
    read), and the outputs."""
    n = (case["NX"] - 2) * (case["NY"] - 2) * (case["NZ"] - 2)
    N = case["NX"] * case["NY"] * case["NZ"]
    pop = 216 if case["storage"] == "f32" else 108
    kind, T = case["kind"], case["steps"]
    if kind == "step":
        per, out, flops = 2 * pop, 20 * N, 450
    elif kind == "granular":  # the moment planes are the launchers' interface
        per, out, flops = 2 * pop + 2 * 48, 20 * N, 450
    elif kind == "restart":
        per, out, flops = 2 * pop, 4 * 216 * N, 450
    else:
        per, out, flops = 2 * pop + 48 + 2 * 216 + 48, (12 if kind == "adjoint" else 0) * N, 450 + 900
    return {"bytes": float(T * per * n + out), "flops": float(T * flops * n)}


# ---------------------------------------------------------------- float64

W = [8 / 27 if q == 0 else 2 / 27 if q == 1 else 1 / 54 if q == 2 else 1 / 216
     for q in (CX[i] ** 2 + CY[i] ** 2 + CZ[i] ** 2 for i in range(Q))]
B0 = [-10 / 27 if i == 0 else W[i] for i in range(Q)]


def _feq(i, rho, u):
    cu = CX[i] * u[0] + CY[i] * u[1] + CZ[i] * u[2]
    usq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
    return W[i] * rho * (1 + 4.5 * cu * cu - 1.5 * usq + 3 * cu + cu * (4.5 * cu * cu - 4.5 * usq))


def _fneq(i, p, u):
    """Regularised non-equilibrium part of direction i; p: xx, xy, yy, yz, zz, xz."""
    x, y, z = CX[i], CY[i], CZ[i]
    pxx, pxy, pyy, pyz, pzz, pxz = p
    a2 = (pxx * (x * x - 1 / 3) + 2 * pxy * x * y + pyy * (y * y - 1 / 3) + 2 * pyz * y * z + pzz * (z * z - 1 / 3)
          + 2 * pxz * x * z)
    a3 = 0.0
    for h, v in ((x * x * y - y / 3, lambda: pxx * u[1] + 2 * pxy * u[0]),
                 (x * x * z - z / 3, lambda: pxx * u[2] + 2 * pxz * u[0]),
                 (x * y * y - x / 3, lambda: pyy * u[0] + 2 * pxy * u[1]),
                 (x * z * z - x / 3, lambda: pzz * u[0] + 2 * pxz * u[2]),
                 (y * y * z - z / 3, lambda: pyy * u[2] + 2 * pyz * u[1]),
                 (y * z * z - y / 3, lambda: pzz * u[1] + 2 * pyz * u[2]),
                 (2 * x * y * z, lambda: pxy * u[2] + pxz * u[1] + pyz * u[0])):
        if h:
            a3 = a3 + h * v()
    return W[i] * (4.5 * a2 + 13.5 * a3)


def _moments(fr, fb):
    """Densities, velocity, non-equilibrium stress of [27] lists of arrays."""
    rr, rb = sum(fr), sum(fb)
    rho = rr + rb
    j = [0.0, 0.0, 0.0]
    s = [0.0] * 6
    for i in range(Q):
        g = fr[i] + fb[i]
        x, y, z = CX[i], CY[i], CZ[i]
        for k, c in enumerate((x, y, z)):
            if c:
                j[k] = j[k] + c * g
        for k, h in enumerate((x * x - 1 / 3, x * y, y * y - 1 / 3, y * z, z * z - 1 / 3, x * z)):
            if h:
                s[k] = s[k] + h * g
    u = [v / rho for v in j]
    p = [s[0] - rho * u[0] * u[0], s[1] - rho * u[0] * u[1], s[2] - rho * u[1] * u[1], s[3] - rho * u[1] * u[2],
         s[4] - rho * u[2] * u[2], s[5] - rho * u[0] * u[2]]
    return rr, rb, u, p


def _splitmix(x):
    x = x + np.uint64(0x9E3779B97F4A7C15)
    x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return x ^ (x >> np.uint64(31))


class _Model:
    """The step in float64 on interior arrays [NZ-2][NY-2][NX-2]; `sigma`,
    `tau` and the profile coefficients `c` may carry gradients."""

    def __init__(self, case, seed, sigma=None, tau=None, c=None):
        p = _parameters(case, seed)
        self.case, self.dev = case, _device()
        self.shape = (case["NZ"], case["NY"], case["NX"])
        self.boundary, self.seed, self.noise = case["boundary"], np.uint64(p["seed"]), p["inlet_noise"]
        f32 = np.float32
        self.tau = float(f32(p["tau"])) if tau is None else tau
        self.sigma = float(f32(p["sigma"])) if sigma is None else sigma
        self.beta = float(f32(p["beta_recolor"]))
        self.t = 0
        NX, NZ = case["NX"], case["NZ"]
        dx = np.arange(NX, dtype=f32) - f32(NX - 1) / f32(2)
        dz = np.arange(NZ, dtype=f32) - f32(NZ - 1) / f32(2)
        r2 = (dx * dx)[None, :] + (dz * dz)[:, None]
        inner = np.zeros((NZ, NX), bool)
        inner[1:-1, 1:-1] = True
        self.inner = inner
        self.jet = torch.from_numpy((r2 <= f32(p["jet_radius"]) ** 2) & inner).to(self.dev)
        self.bins = torch.from_numpy(np.sqrt(r2).astype(np.int64)).to(self.dev)
        self.r = torch.from_numpy(np.sqrt(r2).astype(np.float64)).to(self.dev)
        self.dx = torch.from_numpy(dx.astype(np.float64)).to(self.dev)
        self.dz = torch.from_numpy(dz.astype(np.float64)).to(self.dev)
        self.velocity = float(f32(p["jet_velocity"]))
        self.profile = torch.ones((NZ, NX), dtype=torch.float64, device=self.dev)
        if c is not None:
            from torch.special import bessel_j0

            for k in range(len(c)):
                a = _bessel_zero(k)
                self.profile = self.profile + c[k] * bessel_j0(a * self.r / p["jet_radius"])

    def start(self, F):
        """State of equilibrium populations of the host fields F."""
        full = [torch.from_numpy(np.asarray(v)).to(self.dev).double().reshape(self.shape) for v in F]
        rr, rb, *u = [v[1:-1, 1:-1, 1:-1] for v in full]
        self.full = full
        fr = [_feq(i, rr, u) for i in range(Q)]
        fb = [_feq(i, rb, u) for i in range(Q)]
        psi = (full[0] - full[1]) / (full[0] + full[1])
        out = [v[:, -1, :].clone() for v in full]
        return fr, fb, psi, out

    def _psi_full(self, inner, ghosts):
        if self.boundary == "periodic":
            for d in range(3):
                n = inner.shape[d]
                inner = torch.cat([inner.narrow(d, n - 1, 1), inner, inner.narrow(d, 0, 1)], d)
            return inner
        core = torch.cat([ghosts[1:-1, 1:-1, :1], inner, ghosts[1:-1, 1:-1, -1:]], 2)
        core = torch.cat([ghosts[1:-1, :1], core, ghosts[1:-1, -1:]], 1)
        return torch.cat([ghosts[:1], core, ghosts[-1:]], 0)

    def step(self, fr, fb, psi, out):
        """One step: (moments of the state, next state)."""
        NZ, NY, NX = self.shape
        rr, rb, u, p = _moments(fr, fb)
        rho = rr + rb
        oms = 1 - 1 / self.tau
        P = self._psi_full((rr - rb) / rho, psi)
        g = [0.0, 0.0, 0.0]
        for i in range(1, Q):
            v = W[i] * P[1 + CZ[i]:NZ - 1 + CZ[i], 1 + CY[i]:NY - 1 + CY[i], 1 + CX[i]:NX - 1 + CX[i]]
            for k, c in enumerate((CX[i], CY[i], CZ[i])):
                if c:
                    g[k] = g[k] + 3 * c * v
        F2 = g[0] ** 2 + g[1] ** 2 + g[2] ** 2
        interface = 4 * rr * rb / rho ** 2 > 1e-4
        safe = torch.where(interface & (F2 > 0), F2, torch.ones_like(F2))
        absF = torch.where(interface & (F2 > 0), safe.sqrt(), torch.zeros_like(F2))
        has = absF > 1e-4
        inv = torch.where(has, 1 / safe.sqrt(), torch.zeros_like(F2))
        Ah = self.sigma * (9 / 8) / self.tau
        aR, aB = rr / rho, rb / rho
        amp = self.beta * rr * rb / rho
        post = []
        for i in range(Q):
            fc = CX[i] * g[0] + CY[i] * g[1] + CZ[i] * g[2]
            v = _feq(i, rho, u) + oms * _fneq(i, p, u) + Ah * absF * (W[i] * (fc * inv) ** 2 - B0[i])
            n2 = CX[i] ** 2 + CY[i] ** 2 + CZ[i] ** 2
            d = amp * W[i] * fc * inv / math.sqrt(n2) if n2 else 0.0
            post.append((aR * v + d, aB * v - d))
        if self.boundary == "jet":
            inlet, outlet, psi, out = self._ghosts(rr, rb, u, p, psi, out)
        new = ([], [])
        for i in range(Q):
            for c in range(2):
                v = torch.roll(post[i][c], (CZ[i], CX[i]), (0, 2))
                if self.boundary == "periodic":
                    v = torch.roll(v, CY[i], 1)
                elif CY[i] == 1:
                    edge = (fr, fb)[c][i][:, :1]
                    if self.boundary == "jet":
                        edge = self._delivered(inlet[i][c], i, self.jet, edge)
                    v = torch.cat([edge, v[:, :-1]], 1)
                elif CY[i] == -1:
                    edge = (fr, fb)[c][i][:, -1:]
                    if self.boundary == "jet":
                        edge = self._delivered(outlet[i][c], i, None, edge)
                    v = torch.cat([v[:, 1:], edge], 1)
                new[c].append(v)
        self.t += 1
        return (rr, rb, u, p), (new[0], new[1], psi, out)

    def _delivered(self, value, i, mask, kept):
        """Values [NZ-2][NX-2] of the interior columns delivered to (x+cx, z+cz)."""
        NZ, _, NX = self.shape
        given = torch.ones((NZ - 2, NX - 2), dtype=torch.bool, device=self.dev) if mask is None else mask[1:-1, 1:-1]
        pad = torch.nn.functional.pad
        v, m = pad(value, (1, 1, 1, 1)), pad(given, (1, 1, 1, 1))
        at = (slice(1 - CZ[i], NZ - 1 - CZ[i]), slice(1 - CX[i], NX - 1 - CX[i]))
        return torch.where(m[at].unsqueeze(1), v[at].unsqueeze(1), kept)

    def _ghosts(self, rr, rb, u, p, psi, out):
        NZ, NY, NX = self.shape
        oms = 1 - 1 / self.tau
        vel = self.velocity * self.profile
        if self.noise:
            with np.errstate(over="ignore"):
                x, z = np.meshgrid(np.arange(NX, dtype=np.uint64), np.arange(NZ, dtype=np.uint64))
                h = _splitmix(np.uint64(0x1A1E7) ^ np.uint64(self.t) ^ _splitmix(x ^ _splitmix(z)))
                h = _splitmix(self.seed ^ h)
            noise = 1 + (2 * ((h >> np.uint64(40)).astype(np.float64) / 2 ** 24) - 1) * float(np.float32(self.noise))
            vel = vel * torch.from_numpy(noise).to(self.dev)
        vel = vel[1:-1, 1:-1]
        zero, one = torch.zeros_like(vel), torch.ones_like(vel)
        first = [v[:, 0] for v in u], [v[:, 0] for v in p]
        inlet = {}
        for i in range(Q):
            if CY[i] == 1:
                v = _feq(i, one, (zero, vel, zero)) + oms * _fneq(i, first[1], first[0])
                inlet[i] = (zero, v)
        uc = u[1][:, -1].clamp(0, 1)
        new = []
        for b, f in zip(out, (rr, rb, *u)):
            b_in = b[1:-1, 1:-1]
            new.append(b_in - uc * (b_in - f[:, -1]))
        B = new
        rho = B[0] + B[1]
        last = [v[:, -1] for v in u], [v[:, -1] for v in p]
        outlet = {}
        for i in range(Q):
            if CY[i] == -1:
                v = _feq(i, rho, B[2:]) + oms * _fneq(i, last[1], last[0])
                outlet[i] = (B[0] / rho * v, B[1] / rho * v)

        def put(plane, inside):
            v = torch.cat([plane[1:-1, :1], inside, plane[1:-1, -1:]], 1)
            return torch.cat([plane[:1], v, plane[-1:]], 0)

        out = [put(b, n) for b, n in zip(out, new)]
        m = self.jet[1:-1, 1:-1].double()
        psi = torch.cat([put(psi[:, 0], 1 - 2 * m).unsqueeze(1), psi[:, 1:-1],
                         put(psi[:, -1], (B[0] - B[1]) / rho).unsqueeze(1)], 1)
        return inlet, outlet, psi, out


def _bessel_zero(k):
    """k-th zero of J0 (from 0), by bisection around McMahon's estimate."""
    lo, hi = (k + 0.75) * math.pi - 0.3, (k + 0.75) * math.pi + 0.3
    j0 = lambda v: float(torch.special.bessel_j0(torch.tensor(v, dtype=torch.float64)))  # noqa: E731
    for _ in range(80):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if (j0(lo) > 0) == (j0(mid) > 0) else (lo, mid)
    return 0.5 * (lo + hi)


def exact(case, seed):
    n = case["NX"] * case["NY"] * case["NZ"]
    if n * case["steps"] > (45e6 if case["kind"] in ("adjoint", "jetgrad") else 140e6):
        return None  # over about 20 seconds
    F = _fields(case, seed)
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed, F)
    if case["kind"] == "jetgrad":
        return _exact_jetgrad(case, seed, F)
    with torch.no_grad():
        return _exact_run(case, seed, F)


def _exact_run(case, seed, F):
    M = _Model(case, seed)
    NZ, NY, NX = M.shape
    state = M.start(F)
    nb = NX // 2
    sums = torch.zeros((5, NY, nb), dtype=torch.float64, device=M.dev)
    for _ in range(case["steps"]):
        (rr, rb, u, p), state = M.step(*state)
        if case["stats"]:
            _add_radial(M, sums, u)
    if case["kind"] == "restart":
        pad = torch.nn.functional.pad
        flat = [torch.stack([pad(v, (1, 1, 1, 1, 1, 1)) for v in f]).reshape(-1).cpu().numpy() for f in state[:2]]
        return {"fr": flat[0], "fb": flat[1], "finite": None}
    fields = {}
    for k, (name, v) in enumerate(zip(FIELDS, (rr, rb, *u))):
        w = M.full[k].clone()
        w[1:-1, 1:-1, 1:-1] = v
        if case["boundary"] == "jet":
            w[:, -1, :] = state[3][k]
            if k < 2:
                m = M.jet.double()
                inner = torch.from_numpy(M.inner).to(M.dev)
                w[:, 0, :] = torch.where(inner, m if k else 1 - m, w[:, 0, :])
        fields[name] = w.reshape(-1).cpu().numpy()
    res = {"fields": fields}
    if case["stats"]:
        bins = M.bins[1:-1, 1:-1]
        cols = torch.bincount(bins.reshape(-1), minlength=nb)[:nb].clamp(min=1).double()
        mean = sums / (cols * case["steps"])
        res["radial"] = {k: mean[i].reshape(-1).cpu().numpy() for i, k in enumerate(RADIAL)}
    if case["boundary"] == "periodic":
        res["mass"] = np.array([float(sum(f.sum() for f in fc)) for fc in state[:2]])
    return res


def _add_radial(M, sums, u):
    nb = sums.shape[2]
    dx, dz, r = M.dx[1:-1].view(1, -1), M.dz[1:-1].view(-1, 1), M.r[1:-1, 1:-1]
    safe = torch.where(r > 1e-12, r, torch.ones_like(r))
    ur = torch.where((r > 1e-12).unsqueeze(1), (u[0] * dx.unsqueeze(1) + u[2] * dz.unsqueeze(1)) / safe.unsqueeze(1),
                     torch.zeros_like(u[0]))
    bins = M.bins[1:-1, 1:-1].clamp(max=nb).unsqueeze(1).expand_as(ur)
    rows = torch.arange(ur.shape[1], device=M.dev).view(1, -1, 1)
    at = (rows * (nb + 1) + bins).reshape(-1)
    uy = u[1]
    for k, v in enumerate((uy, uy * uy, ur, ur * ur, ur * uy)):
        s = torch.zeros(ur.shape[1] * (nb + 1), dtype=torch.float64, device=M.dev).index_add_(0, at, v.reshape(-1))
        sums[k, 1:-1] += s.view(-1, nb + 1)[:, :nb]


def _unpack(flat, fixed):
    return list(flat[0]), list(flat[1]), flat[2] if fixed is None else fixed, list(flat[3])


def _reverse(M, state0, steps, last, source):
    """Reverse sweep by autograd, one step at a time.  `last(state)`: the final
    term of J or None; `source(t, moments)`: the term of step t or None.
    Returns J and the gradient of the stacked first state."""
    pack = lambda s: (torch.stack(s[0]), torch.stack(s[1]), s[2], torch.stack(s[3]))  # noqa: E731
    kept = [pack(state0)]
    J = 0.0
    with torch.no_grad():
        for t in range(steps):
            m, s = M.step(*_unpack(kept[-1], None))
            kept.append(pack(s))
    leaf = [v.detach().requires_grad_(True) for v in kept[-1]]
    grads = [torch.zeros_like(v) for v in leaf]
    if last is not None:
        j = last(_unpack(leaf, None))
        J += float(j.detach())
        grads = [torch.zeros_like(v) if g is None else g
                 for v, g in zip(leaf, torch.autograd.grad(j, leaf, allow_unused=True))]
    for t in reversed(range(steps)):
        M.t = t
        leaf = [v.detach().requires_grad_(True) for v in kept[t]]
        with torch.enable_grad():
            m, s = M.step(*_unpack(leaf, None))
            total = sum((a * b).sum() for a, b in zip(pack(s), grads))
            j = source(t, m)
            if j is not None:
                J += float(j.detach())
                total = total + j
        wanted = leaf + M.parameters
        got = torch.autograd.grad(total, wanted, allow_unused=True, retain_graph=True)
        grads = [torch.zeros_like(v) if g is None else g for v, g in zip(leaf, got)]
        for k, g in enumerate(got[len(leaf):]):
            if g is not None:
                M.gradients[k] = M.gradients[k] + g
        kept[t + 1] = None
        del m, s, total, got
    return J, grads


def _exact_adjoint(case, seed, F):
    probe = _Model(case, seed)
    dev = probe.dev
    sigma = torch.tensor(probe.sigma, dtype=torch.float64, device=dev, requires_grad=True)
    tau = torch.tensor(probe.tau, dtype=torch.float64, device=dev, requires_grad=True)
    M = _Model(case, seed, sigma=sigma, tau=tau)
    M.parameters, M.gradients = [sigma, tau], [0.0, 0.0]
    f32 = [np.asarray(v) for v in F]
    target = ((f32[0] - f32[1]) / (f32[0] + f32[1])).reshape(M.shape)[1:-1, 1:-1, 1:-1]
    target = torch.from_numpy(np.ascontiguousarray(target)).to(dev).double()

    def last(s):
        rr, rb = sum(s[0]), sum(s[1])
        return (((rr - rb) / (rr + rb) - target) ** 2).sum()

    with torch.no_grad():
        state = M.start(F)
    J, g = _reverse(M, state, case["steps"], last, lambda t, m: None)
    u = [M.full[2 + k][1:-1, 1:-1, 1:-1].clone().requires_grad_(True) for k in range(3)]
    rho = [M.full[k][1:-1, 1:-1, 1:-1] for k in range(2)]
    dot = sum((_feq(i, rho[c], u) * g[c][i]).sum() for i in range(Q) for c in range(2))
    du = torch.autograd.grad(dot, u)
    pad = torch.nn.functional.pad
    return {"J": J, "dJ_dsigma": float(M.gradients[0]), "dJ_dtau": float(M.gradients[1]),
            "dJ_du0": torch.stack([pad(v, (1, 1, 1, 1, 1, 1)).reshape(-1) for v in du]).cpu().numpy()}


def _exact_jetgrad(case, seed, F):
    c = torch.zeros(8, dtype=torch.float64, device=_device())
    c[:3] = torch.tensor([float(np.float32(v)) for v in (0.1, -0.05, 0.02)], dtype=torch.float64)
    c.requires_grad_(True)
    M = _Model(case, seed, c=c)
    M.parameters, M.gradients = [c], [0.0]
    t0, y0 = _window(case)
    with torch.no_grad():
        state = M.start(F)

    def source(t, m):
        return 0.5 * (m[2][1][:, y0 - 1:] ** 2).sum() if t >= t0 else None

    J, _ = _reverse(M, state, case["steps"], None, source)
    return {"J": J, "dJ_dc": M.gradients[0].cpu().numpy()}
