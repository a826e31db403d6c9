"""The framework's measured cases: its public entry points over the range that its users run.

``listed()`` names them, ``draw(rng)`` gives more of the same ranges, ``prepare`` makes what a
caller holds before a call (the model, its handle, the inputs), ``run`` is one pass, ``work`` the
bytes and operations that the pass cannot do without and ``exact`` its outputs in plain 64-bit
torch.  Seven kinds of pass:

    fbc       ``Solver.FBC``: the friction solve of one time step on host fault arrays
    apply     ``eqc_apply_K_device``: y = K x on device vectors, FP64 or FP32
    solve     ``Solver.qs_solve``: one quasi-static solve on host arrays, plain FP64
    qs, dyn   ``Solver.init``, ``Solver.run``, ``Solver.state``: time steps of one regime from the
              model's initial state, then the state read back (into page-locked memory)
    ensemble  ``Ensemble.run``: the same for several uneven models, one graph launch per step
    grad      ``Solver.guess_grad``: gradient of the learned guess's loss over one batch
"""
import ctypes
import math

import numpy as np
import torch

from eqcycle_gb300 import (EQC_FP64, EQC_GUESS_EXTRAPOLATE, EQC_GUESS_PREVIOUS, EQC_MIXED, EQC_PC_AMG, EQC_PC_JACOBI,
                           Ensemble, Solver, preset, set_parameters, structured_parameters)
from eqcycle_gb300 import _lib

GRID_X, GRID_Y = 121, 61      # the learned guess's output grid
HIDDEN, CHANNELS, LAYERS = 512, 64, 4


def listed():
    return [
        # the smallest call: one step's friction solve for a host code that keeps its own time loop
        {"name": "fbc_961", "kind": "fbc", "depth": 240, "normal": 480, "damage": 2},
        # a stiffness apply on a small mesh of odd sizes: launch latency and ragged tiles
        {"name": "apply_f32_75x131", "kind": "apply", "depth": 75, "normal": 131, "damage": 1, "fp64": False},
        # the stiffness apply of the plain method on the bench workload
        {"name": "apply_f64_dz480", "kind": "apply", "depth": 240, "normal": 480, "damage": 2, "fp64": True},
        # cg! replaced by itself in the reference's loop, on its own kind of model (a damage rectangle)
        {"name": "solve_90x60", "kind": "solve", "depth": 90, "normal": 60, "damage": 1},
        # interseismic steps of the small homogeneous model, default settings: all launch latency
        {"name": "qs_mixed_homog48", "kind": "qs", "depth": 48, "normal": 48, "damage": 0, "mixed": True,
         "tuned": False, "steps": 12},
        # interseismic steps of the bench workload with the settings that the autotuner settles on
        {"name": "qs_mixed_dz480", "kind": "qs", "depth": 240, "normal": 480, "damage": 2, "mixed": True, "tuned": True,
         "steps": 6},
        # the same on the refined model, the largest that the workloads have
        {"name": "qs_mixed_dz960", "kind": "qs", "depth": 480, "normal": 960, "damage": 2, "mixed": True, "tuned": True,
         "steps": 3},
        # interseismic steps of the plain FP64 method (the default precision), default settings
        {"name": "qs_fp64_dz240", "kind": "qs", "depth": 120, "normal": 240, "damage": 2, "mixed": False,
         "tuned": False, "steps": 3},
        # a rupture of the bench workload: Newmark steps with the fault sliding
        {"name": "dyn_mixed_dz480", "kind": "dyn", "depth": 240, "normal": 480, "damage": 2, "mixed": True,
         "tuned": True, "steps": 200},
        # a rupture by the plain method on a mesh of odd sizes with a damage rectangle
        {"name": "dyn_fp64_61x95", "kind": "dyn", "depth": 61, "normal": 95, "damage": 1, "mixed": False,
         "tuned": False, "steps": 100},
        # an ensemble of uneven damage-zone models, quasi-static
        {"name": "ensemble_8", "kind": "ensemble", "members": 8, "nmin": 80, "nmax": 240, "steps": 4},
        # one training batch of the learned initial guess, forward and backward
        {"name": "grad_256", "kind": "grad", "depth": 240, "normal": 8, "damage": 0, "pairs": 256},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fbc", "apply", "apply", "solve", "qs", "qs", "qs", "dyn", "dyn", "ensemble", "grad"])
    damage = rng.choice([0, 1, 2])
    if kind == "fbc":
        return {"kind": kind, "depth": _log(rng, 24, 480), "normal": _log(rng, 24, 480), "damage": damage}
    if kind == "apply":
        depth = _log(rng, 24, 480)
        return {"kind": kind, "depth": depth, "normal": int(depth * rng.uniform(1.0, 2.0)), "damage": damage,
                "fp64": rng.random() < 0.5}
    if kind == "solve":
        depth = _log(rng, 24, 120)
        return {"kind": kind, "depth": depth, "normal": int(depth * rng.uniform(0.66, 2.0)), "damage": damage}
    if kind == "qs":
        mixed = rng.random() < 0.75
        depth = _log(rng, 24, 480 if mixed else 120)
        return {"kind": kind, "depth": depth, "normal": int(depth * rng.uniform(1.0, 2.0)), "damage": damage,
                "mixed": mixed, "tuned": mixed and rng.random() < 0.5, "steps": rng.randint(2, 3 if depth > 240 else 6)}
    if kind == "dyn":
        mixed = rng.random() < 0.75
        depth = _log(rng, 24, 400 if mixed else 120)
        return {"kind": kind, "depth": depth, "normal": int(depth * rng.uniform(1.0, 2.0)), "damage": damage,
                "mixed": mixed, "tuned": mixed and rng.random() < 0.5, "steps": rng.randint(40, 200)}
    if kind == "ensemble":
        return {"kind": kind, "members": rng.randint(3, 10), "nmin": 48, "nmax": _log(rng, 120, 300),
                "steps": rng.randint(2, 5)}
    return {"kind": kind, "depth": _log(rng, 48, 300), "normal": 8, "damage": 0, "pairs": _log(rng, 16, 400)}


# ---------------------------------------------------------------------------- models and inputs
def _config(case, seed):
    """A model of the damage-zone family over 24 km of depth, elements about square, seeded noise."""
    nx, ny = case["depth"], case["normal"]
    cfg = preset("dz480", seed=seed).replace(NelX=nx, NelY=ny, LY=24e3 * ny / nx, damage=case["damage"])
    return cfg.replace(ThickX=12e3, ThickY=600.0) if case["damage"] == 1 else cfg


def _members(case, seed):
    """Uneven damage-zone models: mesh, zone width, velocity reduction and Dc drawn per member."""
    rng = np.random.default_rng(seed)
    size = np.random.default_rng(case["members"])      # the meshes belong to the case, not to the seed
    out = []
    for k in range(case["members"]):
        n = int(size.integers(case["nmin"], case["nmax"] + 1))
        w = float(rng.uniform(100.0, 2000.0))
        out.append(preset("dz%d" % n, seed=seed + 1000 + k).replace(
            trap_w0=w, trap_w1=0.4 * w, vs2=(1.0 - float(rng.uniform(0.1, 0.6))) * 3464.0,
            Dc=float(np.exp(rng.uniform(np.log(4e-3), np.log(16e-3))))))
    return out


def _steady_dt(P):
    """The step dtevol! takes for steady sliding at the initial rate."""
    nfbc = len(set(P.iarray.FltIglobBC.tolist()) & set(P.iarray.iFlt.tolist()))
    return min(float(np.min(P.farray.XiLf[nfbc:])) / P.cfg.V_init, 50.0 * 86400)


def _options(case):
    """The two methods.  The CG tolerance is that of the package's own smoke run, two digits below
    the benchmark's: the solver's stopping error then lies below what the outputs are compared to."""
    if not case["mixed"]:
        return dict(precision=EQC_FP64, guess=EQC_GUESS_PREVIOUS, cg_tol=1e-10)
    opt = dict(precision=EQC_MIXED, guess=EQC_GUESS_EXTRAPOLATE, cg_tol=1e-10)
    return dict(opt, mg_degree=4, mg_degree_coarse=1, apply_variant=0, reliable_delta=1e-4) if case["tuned"] else opt


def _vector(seed, ny, nx):
    """A displacement-like node field: a few smooth modes and 1 % noise."""
    g = torch.Generator().manual_seed(seed)
    c = torch.randn(4, generator=g, dtype=torch.float64)
    yy = torch.linspace(0, 1, ny, dtype=torch.float64)[:, None]
    xx = torch.linspace(0, 1, nx, dtype=torch.float64)[None, :]
    v = sum(float(c[k]) * torch.cos((k + 1) * 3.0 * xx + k) * torch.exp(-(k + 1) * yy) for k in range(4))
    return v + 0.01 * torch.randn(ny, nx, generator=g, dtype=torch.float64)


def _fault_slip(seed, n):
    """Fault displacement in m: locked above, creeping below, seeded bumps."""
    rng = np.random.default_rng(seed)
    z = np.linspace(0, 1, n)
    return 1e-2 * (1 - z) + sum(rng.normal(0, 1e-3) * np.sin((k + 1) * np.pi * z) for k in range(6))


def _friction_inputs(case, seed, P):
    """Slip rates from locked to seismic, their steady-like state, and the stress-free velocity."""
    rng = np.random.default_rng(seed)
    n = P.int_.FltNglob
    z = np.linspace(0, 1, n)
    lv = -9 + 8.5 * np.exp(-((z - rng.uniform(0.3, 0.7)) / 0.15) ** 2) + rng.normal(0, 0.05, n)
    Vf = 10.0 ** lv
    psi = np.log(P.farray.Vo / Vf) * 0.9 + rng.normal(0, 0.02, n)
    tau = P.farray.Seff * (P.farray.fo + P.farray.cca * np.log(Vf / P.farray.Vo) + P.farray.ccb * psi)
    free = Vf + (tau - P.farray.tauo) / P.farray.FltZ
    return psi, Vf, free


def _weights(seed, nf):
    """Network parameters as one float32 vector: convolutions, fc1, fc2, each weights then biases."""
    g = torch.Generator().manual_seed(seed)
    t = nf
    shapes = []
    for k in range(LAYERS):
        shapes.append((CHANNELS, 2 if k == 0 else CHANNELS, 5))
        t = (t - 1) // 2 + 1
    shapes += [(HIDDEN, CHANNELS * t), (GRID_X * GRID_Y, HIDDEN)]
    parts = []
    for s in shapes:
        lim = math.sqrt(6.0 / math.prod(s[1:]))
        parts.append((torch.rand(s, generator=g) * 2 - 1) * lim)
        parts.append(torch.randn(s[0], generator=g) * 0.01)
    return parts


def _pairs(seed, n, nf):
    g = torch.Generator().manual_seed(seed + 1)
    x = torch.randn(n, 2, nf, generator=g).cumsum(2) / math.sqrt(nf)
    y = torch.randn(n, GRID_Y, GRID_X, generator=g).cumsum(2) / GRID_X
    return x.reshape(n, -1).numpy(), y.reshape(n, -1).numpy()


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


def _stepper(case, cfg):
    P = structured_parameters(cfg)
    s = Solver(P, **_options(case))
    out = {k: _pinned(P.int_.nglob if k in ("d", "v", "a") else P.int_.FltNglob)
           for k in (("d", "v", "psi", "tau") if case["kind"] != "dyn" else ("d", "v", "a", "psi", "tau"))}
    return {"solver": s, "out": out, "V": 5e-2 if case["kind"] == "dyn" else cfg.V_init, "dt": _steady_dt(P)}


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("qs", "dyn"):
        return dict(_stepper(case, _config(case, seed)), case=case)
    if kind == "ensemble":
        mem = [_stepper(dict(case, mixed=True, tuned=False), c) for c in _members(case, seed)]
        return {"case": case, "members": mem, "ensemble": Ensemble([m["solver"] for m in mem])}
    P = structured_parameters(_config(case, seed))
    if kind == "apply":
        s = Solver(P, precond=EQC_PC_JACOBI)
        nx, ny, ld = s.layout()
        x = torch.zeros(ny, ld, dtype=torch.float64)
        x[:, :nx] = _vector(seed, ny, nx)
        x = x.to("cuda", torch.float64 if case["fp64"] else torch.float32)
        return {"case": case, "solver": s, "x": x, "y": torch.zeros_like(x)}
    if kind == "fbc":
        s = Solver(P, precond=EQC_PC_JACOBI)
        psi, Vf, free = _friction_inputs(case, seed, P)
        return {"case": case, "solver": s, "psi": psi, "Vf": Vf, "free": free, "dt": P.float_.dt0}
    if kind == "solve":
        s = Solver(P, precision=EQC_FP64, precond=EQC_PC_AMG)
        return {"case": case, "solver": s, "F": _fault_slip(seed, P.int_.FltNglob), "guess": np.zeros(P.int_.nglob)}
    s = Solver(P, precond=EQC_PC_JACOBI)
    s.set_guess_params(torch.cat([w.reshape(-1) for w in _weights(seed, P.int_.FltNglob)]).numpy())
    x, y = _pairs(seed, case["pairs"], P.int_.FltNglob)
    return {"case": case, "solver": s, "x": x, "y": y}


# ---------------------------------------------------------------------------- one pass
def _start(m, dyn):
    m["solver"].init(m["V"])
    m["solver"].set_scalar("isolver", 2) if dyn else m["solver"].set_scalar("dt", m["dt"])


def _read(m):
    return {k: m["solver"].state(k, out=v) for k, v in m["out"].items()}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("qs", "dyn"):
        _start(state, kind == "dyn")
        state["solver"].run(case["steps"])
        return dict(_read(state), time=state["solver"].result("time_"))
    if kind == "ensemble":
        for m in state["members"]:
            _start(m, False)
        state["ensemble"].run(case["steps"])
        return [_read(m) for m in state["members"]]
    s = state["solver"]
    if kind == "apply":
        x, y = state["x"], state["y"]
        _lib.check(_lib.lib().eqc_apply_K_device(s.h, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(y.data_ptr()),
                                                 0 if case["fp64"] else 1), s.h)
        return y
    if kind == "fbc":
        z = np.zeros(s.Nf)
        return s.FBC(z, z, z, z, z, z, state["psi"], state["Vf"], state["free"], state["dt"])
    if kind == "solve":
        return s.qs_solve(state["F"], state["guess"], tol=1e-10)[0]
    return s.guess_grad(state["x"], state["y"])


# ---------------------------------------------------------------------------- bounds
def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        size = np.random.default_rng(case["members"])
        total = {"bytes": 0.0, "flops": 0.0}
        for _ in range(case["members"]):
            n = int(size.integers(case["nmin"], case["nmax"] + 1))
            w = work({"kind": "qs", "depth": n // 2, "normal": n, "mixed": True, "steps": case["steps"]})
            total = {k: total[k] + w[k] for k in total}
        return total
    nel = case["depth"] * case["normal"]
    nf = 4 * case["depth"] + 1
    n = nf * (4 * case["normal"] + 1)
    apply_flops = 10 * (2 * 2 * 25 + 5) * nel           # five lines each way, two 5-point contractions a line
    if kind == "fbc":                                    # six results, three states, nine parameters
        return {"bytes": 8.0 * 18 * nf, "flops": 400.0 * nf}
    if kind == "apply":
        return {"bytes": (8 if case["fp64"] else 4) * (2.0 * n + 25 * nel), "flops": float(apply_flops)}
    if kind == "solve":                                  # the guess in, the solution out, one apply's data
        return {"bytes": 8.0 * (2 * n + 25 * nel), "flops": float(apply_flops)}
    if kind == "qs":                                     # two solves a step, each at least one apply's data
        return {"bytes": case["steps"] * 2.0 * (8 * 3 * n + (4 if case["mixed"] else 8) * 25 * nel),
                "flops": case["steps"] * 2.0 * apply_flops}
    if kind == "dyn":                                    # d, v, K d or a, 1/M, and the apply's data
        return {"bytes": case["steps"] * (8.0 * 7 * n + (4 if case["mixed"] else 8) * 25 * nel),
                "flops": float(case["steps"] * (apply_flops + 8 * n))}
    t, flops, params = nf, 0.0, 0
    for k in range(LAYERS):
        t = (t - 1) // 2 + 1
        size = CHANNELS * (2 if k == 0 else CHANNELS) * 5
        params += size + CHANNELS
        flops += (4.0 if k == 0 else 6.0) * size * t
    size = HIDDEN * (CHANNELS * t + GRID_X * GRID_Y)
    params += size + HIDDEN + GRID_X * GRID_Y
    return {"bytes": 4.0 * (case["pairs"] * (2 * nf + GRID_X * GRID_Y) + 2 * params),
            "flops": case["pairs"] * (flops + 6.0 * size)}


# ---------------------------------------------------------------------------- the same in 64 bits
_DEV = "cuda" if torch.cuda.is_available() else "cpu"


class _Model:
    """The setup's arrays on the node grid [fault normal, depth] in 64 bits, and the operators."""

    def __init__(self, cfg):
        P = set_parameters(cfg)
        m, f = P.mesh, P.farray
        self.P, self.cfg = P, cfg
        self.ex, self.ey = m.NelX, m.NelY
        self.nx, self.ny = 4 * m.NelX + 1, 4 * m.NelY + 1
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=_DEV)  # noqa: E731
        self.H = t(m.H)
        self.W = t(np.asarray(m.W).transpose(2, 1, 0).reshape(self.ey, self.ex, 5, 5))    # [ey, ex, j, i]
        hx, hy = 0.5 * m.dxe, 0.5 * m.dye
        self.c1, self.c2 = hy / hx, hx / hy
        ids = np.empty((self.ny, self.nx), dtype=np.int64)                                # grid -> reference node
        ig = np.asarray(m.iglob).transpose(2, 1, 0).reshape(self.ey, self.ex, 5, 5) - 1
        for j in range(5):
            for i in range(5):
                ids[j:j + 4 * self.ey - 3:4, i:i + 4 * self.ex - 3:4] = ig[:, :, j, i]
        self.ids = torch.as_tensor(ids, device=_DEV)
        self.M = t(f.M)[self.ids]
        flat = np.empty(ids.size, dtype=np.int64)
        flat[ids.reshape(-1)] = np.arange(ids.size)
        self.left = torch.as_tensor(flat[P.iarray.iBcL - 1], device=_DEV)
        self.top = torch.as_tensor(flat[P.iarray.iBcT - 1], device=_DEV)
        self.cl, self.ct = t(f.BcLC), t(f.BcTC)
        for k in ("fo", "Vo", "xLf", "FltB", "FltZ", "cca", "ccb", "Seff", "tauo", "XiLf"):
            setattr(self, k, t(getattr(f, k)))
        self.creep = torch.zeros(self.nx, dtype=torch.bool, device=_DEV)
        c = flat[P.iarray.FltIglobBC - 1]
        self.creep[torch.as_tensor(c[c < self.nx], device=_DEV)] = True
        self.Vpl = P.float_.Vpl

    def _sum(self, a):
        """Element contributions [ey, ex, j, i] summed at the nodes."""
        y = torch.zeros(self.ny, self.nx, dtype=torch.float64, device=_DEV)
        for j in range(5):
            for i in range(5):
                y[j:j + 4 * self.ey - 3:4, i:i + 4 * self.ex - 3:4] += a[:, :, j, i]
        return y

    def K(self, x):
        u = x.unfold(0, 5, 4).unfold(1, 5, 4).contiguous()                                # [ey, ex, j, i]
        return self._sum(self.c1 * ((self.W * (u @ self.H)) @ self.H.T) +
                         self.c2 * (self.H @ (self.W * (self.H.T @ u))))

    def diag(self):
        H2 = self.H ** 2
        return self._sum(self.c1 * (self.W @ H2.T) + self.c2 * (H2 @ self.W))

    def solve(self, d, tol):
        """d off the fault row with (K d) = 0 there, the fault row given: Jacobi-preconditioned CG."""
        d, dg = d.clone(), self.diag()
        b = torch.zeros_like(d)
        b[0] = d[0]
        b = self.K(b)[1:]
        r = -self.K(d)
        r[0] = 0
        stop = tol * float(b.norm())
        if float(r.norm()) <= stop:
            return d
        z = r / dg
        p, rz = z.clone(), (r * z).sum()
        for it in range(20000):
            q = self.K(p)
            q[0] = 0
            alpha = rz / (p * q).sum()
            d += alpha * p
            r -= alpha * q
            if it % 16 == 15 and float(r.norm()) <= stop:
                break
            z = r / dg
            rz, old = (r * z).sum(), rz
            p = z + (rz / old) * p
        return d

    def out(self, x):
        """A grid field in the reference numbering, on the host."""
        y = torch.empty(x.numel(), dtype=torch.float64, device=_DEV)
        y[self.ids.reshape(-1)] = x.reshape(-1)
        return y.cpu().numpy()

    # friction
    def ids1(self, psi, dt, Vf, small):
        w = Vf.abs() * dt / self.xLf
        lo = torch.exp(psi - w) + self.Vo * dt / self.xLf - 0.5 * self.Vo * Vf.abs() * dt * dt / self.xLf ** 2
        hi = torch.exp(psi - w) + (self.Vo / Vf.abs()) * (1 - torch.exp(-w))
        return torch.log(torch.where(w < small, lo, hi))

    def ids2(self, psi, dt, Vf, Vf1):
        return self.ids1(psi, dt, 0.5 * (Vf + Vf1).abs(), 1e-6)

    def newton(self, tau, psi, free):
        fact = 1 + (self.Vo / 1e10) * torch.exp(-psi)
        eps, scale = 0.001 * self.cca * self.Seff, self.Seff * self.cca
        h = -(self.fo + self.ccb * psi) / self.cca
        tau, V = tau.clone(), torch.zeros_like(tau)
        on = torch.ones_like(tau, dtype=torch.bool)
        for _ in range(1000):
            a, b = torch.exp(h + fact * tau / scale), torch.exp(h - fact * tau / scale)
            V = self.Vo * (a - b)
            delta = (self.FltZ * free - self.FltZ * V + self.tauo - tau) / (1 + self.FltZ * fact * (self.Vo / scale) * (a + b))
            tau = torch.where(on, tau + delta, tau)
            on = on & (delta.abs() > eps)
            if not bool(on.any()):
                break
        return tau, self.Vo * (torch.exp(h + fact * tau / scale) - torch.exp(h - fact * tau / scale))

    def fbc(self, psi, Vf, free, dt):
        p1 = self.ids1(psi, dt, Vf, 1e-5)
        t1, v1 = self.newton(torch.zeros_like(psi), p1, free)
        p2 = self.ids2(psi, dt, Vf, v1)
        t2, v2 = self.newton(t1, p2, free)
        return p1, v1, t1, p2, v2, t2

    def steps(self, V, dyn, dt, n, names):
        d = torch.zeros(self.ny, self.nx, dtype=torch.float64, device=_DEV)
        a, c = torch.zeros_like(d), self.creep
        v = torch.full_like(d, 0.5 * V)
        psi = self.tauo / (self.Seff * self.ccb) - self.fo / self.ccb - (self.cca / self.ccb) * torch.log(
            2 * v[0] / self.Vo)
        v -= 0.5 * self.Vpl
        v[0, c] = 0
        zero, tau = torch.zeros_like(psi), torch.zeros_like(psi)
        t, times, dt0 = 0.0, [], self.P.float_.dt0
        dt = dt0 if dyn else dt
        for _ in range(n):
            t += dt
            times.append(t)
            if dyn:
                pre = v[0].clone()
                d = d + dt * v + 0.5 * dt * dt * a
                v = v + 0.5 * dt * a
                a = -self.K(d)
                a[0, c] = 0
                vf = v.reshape(-1)
                a.view(-1)[self.left] -= self.cl * vf[self.left]
                a.view(-1)[self.top] -= self.ct * vf[self.top]
                _, _, _, p2, _, t2 = self.fbc(psi, 2 * pre + self.Vpl, 2 * v[0] + dt * a[0] / self.M[0], dt)
                psi, tau = torch.where(c, zero, p2), torch.where(c, zero, t2 - self.tauo)
                a[0] -= self.FltB * tau
                a = a / self.M
                v = v + 0.5 * dt * a
                v[0, c] = 0
                a[0, c] = 0
                continue
            pre, V0 = d.clone(), 2 * v[0] + self.Vpl
            Vf, vF = V0, v[0].clone()
            for _ in range(2):
                d[0] = pre[0] + vF * dt
                d = self.solve(d, 1e-12)
                t1 = torch.where(c, zero, -self.K(d)[0] / self.FltB)
                p1 = self.ids1(psi, dt, Vf, 1e-6)
                h, fa = -(self.fo + self.ccb * p1) / self.cca, (t1 + self.tauo) / (self.Seff * self.cca)
                V1 = torch.where(c, zero + self.Vpl, self.Vo * (torch.exp(h + fa) - torch.exp(h - fa)))
                Vf = 0.5 * (V0 + V1)
                vF = 0.5 * (Vf - self.Vpl)
            psi, tau = torch.where(c, zero, p1), t1
            v = (d - pre) / dt
            v[0] = 0.5 * (V1 - self.Vpl)
            d[0, c] = 0
            v[0, c] = 0
            rate = (2 * v[0] + self.Vpl)[~c].abs()
            dt = min(max(min(50.0 * 86400, float((self.XiLf[~c] / rate).min())), dt0), 1.2 * dt)
        got = {"d": self.out(d), "v": self.out(v), "a": self.out(a), "psi": psi.cpu().numpy(), "tau": tau.cpu().numpy()}
        return {k: got[k] for k in names} | {"time": np.array(times)}


def _network(case, seed):
    """Loss and gradients by autograd: bfloat16 weights held in 64 bits, exact products and sums."""
    P = structured_parameters(_config(case, seed))
    nf, n = P.int_.FltNglob, case["pairs"]
    ws = [w.to(torch.bfloat16).double() if k % 2 == 0 else w.double() for k, w in enumerate(_weights(seed, nf))]
    ws = [w.to(_DEV).requires_grad_() for w in ws]
    x, y = (torch.as_tensor(v, device=_DEV).double() for v in _pairs(seed, n, nf))
    h = x.reshape(n, 2, nf)
    F = torch.nn.functional
    for k in range(LAYERS):
        h = F.gelu(F.conv1d(h, ws[2 * k], ws[2 * k + 1], stride=2, padding=2))
    h = F.gelu(h.reshape(n, -1) @ ws[-4].T + ws[-3])
    loss = ((h @ ws[-2].T + ws[-1] - y) ** 2).mean()
    loss.backward()
    return torch.cat([w.grad.reshape(-1) for w in ws]).cpu().numpy(), float(loss)


def exact(case, seed):
    kind = case["kind"]
    if kind == "grad":
        return _network(case, seed)
    if kind == "ensemble":
        return None                                     # members of the qs kind, minutes of plain CG
    if kind == "qs" and 2 * case["steps"] * max(case["depth"], case["normal"]) > 1500:
        return None                                     # the same
    if max(case["depth"], case["normal"]) > 500:
        return None                                     # the host setup and the steps take too long
    m = _Model(_config(case, seed))
    if kind == "apply":
        ld = (m.nx + 7) // 8 * 8
        y = torch.zeros(m.ny, ld, dtype=torch.float64, device=_DEV)
        x = _vector(seed, m.ny, m.nx)
        y[:, :m.nx] = m.K((x if case["fp64"] else x.float().double()).to(_DEV))
        return y
    if kind == "fbc":
        ins = [torch.as_tensor(v, device=_DEV) for v in _friction_inputs(case, seed, m.P)]
        got = m.fbc(*ins, m.P.float_.dt0)
        return tuple(torch.where(m.creep, torch.zeros_like(g), g).cpu().numpy() for g in got)
    if kind == "solve":
        d = torch.zeros(m.ny, m.nx, dtype=torch.float64, device=_DEV)
        d[0] = torch.as_tensor(_fault_slip(seed, m.nx))
        return m.out(m.solve(d, 1e-13))
    V = 5e-2 if kind == "dyn" else m.cfg.V_init
    names = ("d", "v", "psi", "tau") if kind == "qs" else ("d", "v", "a", "psi", "tau")
    return m.steps(V, kind == "dyn", _steady_dt(m.P), case["steps"], names)
