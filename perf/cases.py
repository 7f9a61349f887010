"""Measured cases of the compressible-flow solvers: what a user's program has
this package do, through its public entry points.

A case is a dict of plain values with a "kind":

  step      emg_uniform_step_noalloc on device tensors of the caller: one step
  uniform   GpuSolver: upload an initial state, advance some CFL steps, download
  amr       GpuAmr: CFL steps of a block hierarchy that regrids, then download
  batch     GpuBatch1D: many 1-D Riemann problems to the next output time
  adjoint   DifferentiableSolver: record a run, objective, gradients
  five      GpuFiveSolver: CFL steps of the two-phase system, then download

Every pass returns the whole state that it computes (and the gradients, for the
adjoint). ``exact`` is an independent float64 restatement in plain torch of the
Euler scheme (WENO5-Z/WCNS interpolation, HLLC, positivity limiter, SSP-RK3,
boundary layers, CFL step); the block hierarchy and the two-phase system have no
such restatement here.
"""
import ctypes as C
import math

import numpy as np
import torch

from emergence_b200 import _abi, workloads
from emergence_b200.adjoint import OBJ_ENERGY, OBJ_PRESSURE, DifferentiableSolver
from emergence_b200.amr import GpuAmr
from emergence_b200.batch import GpuBatch1D
from emergence_b200.five import FiveEq, GpuFiveSolver
from emergence_b200.physics import Bc, Euler, FluxMode, Mesh, Nasg, Precision
from emergence_b200.solver import GpuSolver, _c_bcs, _c_eos, _c_mesh

PRECISION = {"f64": Precision.F64, "mixed": Precision.Mixed, "fast": Precision.F64Fast}
MODE = {"weno": FluxMode.Weno, "hybrid": FluxMode.Hybrid}
NG = 6


def listed():
    return [
        # the smallest call: one step of a small patch that lives in the caller's own device memory
        {"name": "step 48x48 f64", "kind": "step", "n0": 48, "n1": 48, "n2": 1, "precision": "f64"},
        # a shock tube between two outputs: launch latency, one line of cells
        {"name": "tube 400 f64", "kind": "uniform", "problem": "blast", "n0": 400, "n1": 1, "n2": 1, "mode": "weno",
         "precision": "f64", "bc": "outflow", "steps": 40},
        # 2-D explosion at the size of the gradient workload's forward run
        {"name": "explosion 512x512 f64", "kind": "uniform", "problem": "blast", "n0": 512, "n1": 512, "n2": 1,
         "mode": "weno", "precision": "f64", "bc": "outflow", "steps": 20},
        # shock running into density waves, hybrid fluxes, a stiffened gas, odd extents, walls and inflow
        {"name": "waves 301x187 hybrid f64", "kind": "uniform", "problem": "waves", "n0": 301, "n1": 187, "n2": 1,
         "mode": "hybrid", "precision": "f64", "bc": "tunnel", "steps": 16},
        # the headline workload: 3-D explosion, bit-exact form
        {"name": "explosion 256^3 f64", "kind": "uniform", "problem": "blast", "n0": 256, "n1": 256, "n2": 256,
         "mode": "weno", "precision": "f64", "bc": "outflow", "steps": 5},
        # ragged 3-D box, fast FP64 form, periodic
        {"name": "explosion 161x127x98 fast", "kind": "uniform", "problem": "blast", "n0": 161, "n1": 127, "n2": 98,
         "mode": "weno", "precision": "fast", "bc": "periodic", "steps": 12},
        # 3-D, FP32 interpolation
        {"name": "explosion 192^3 mixed", "kind": "uniform", "problem": "blast", "n0": 192, "n1": 192, "n2": 192,
         "mode": "weno", "precision": "mixed", "bc": "outflow", "steps": 8},
        # 3-D shock-bubble on three levels with regrids
        {"name": "amr bubble 3d f64", "kind": "amr", "dim": 3, "base": 4, "levels": 3, "precision": "f64",
         "subcycle": False, "steps": 12},
        # 2-D hierarchy: many small launches per step
        {"name": "amr bubble 2d fast", "kind": "amr", "dim": 2, "base": 8, "levels": 4, "precision": "fast",
         "subcycle": False, "steps": 16},
        # a batch of Riemann problems of very different lengths
        {"name": "batch 4096 f64", "kind": "batch", "ninst": 4096, "nmax": 2048, "precision": "f64", "frame": 0.0024},
        # one gradient: forward run with checkpoints, recompute, reverse sweeps
        {"name": "adjoint 192x192", "kind": "adjoint", "n0": 192, "n1": 192, "n2": 1, "objective": "pressure",
         "steps": 16},
        # two-phase shock-bubble
        {"name": "five 96^3 f64", "kind": "five", "n": 96, "precision": "f64", "steps": 10},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "uniform", "uniform", "uniform", "amr", "batch", "adjoint", "five"])
    prec = rng.choice(["f64", "f64", "fast", "mixed"])
    if kind == "step":
        n0 = _log_int(rng, 24, 300)
        return {"kind": kind, "n0": n0, "n1": _log_int(rng, 16, 300), "n2": 1, "precision": prec}
    if kind == "uniform":
        dim = rng.choice([1, 2, 2, 3, 3])
        waves = dim == 2 and rng.random() < 0.4
        if dim == 1:
            n = [_log_int(rng, 64, 20000), 1, 1]
        elif dim == 2:
            n = [_log_int(rng, 48, 900), _log_int(rng, 48, 900), 1]
        else:
            n = [_log_int(rng, 24, 200) for _ in range(3)]
        cells = n[0] * n[1] * n[2]
        steps = max(2, min(40, int(4e7 / cells)))
        return {"kind": kind, "problem": "waves" if waves else "blast", "n0": n[0], "n1": n[1], "n2": n[2],
                "mode": "hybrid" if waves else "weno", "precision": prec,
                "bc": "tunnel" if waves else rng.choice(["outflow", "periodic", "reflect"]), "steps": steps}
    if kind == "amr":
        dim = rng.choice([2, 2, 3])
        return {"kind": kind, "dim": dim, "base": rng.randint(3, 4) if dim == 3 else rng.randint(4, 12),
                "levels": rng.randint(2, 3) if dim == 3 else rng.randint(2, 4), "precision": rng.choice(["f64", "fast"]),
                "subcycle": dim == 2 and rng.random() < 0.4, "steps": rng.randint(4, 10)}
    if kind == "batch":
        return {"kind": kind, "ninst": _log_int(rng, 64, 4096), "nmax": _log_int(rng, 128, 2048), "precision": prec,
                "frame": 0.0024}
    if kind == "adjoint":
        return {"kind": kind, "n0": _log_int(rng, 48, 260), "n1": _log_int(rng, 48, 260), "n2": 1,
                "objective": rng.choice(["pressure", "energy"]), "steps": rng.randint(4, 16)}
    return {"kind": kind, "n": rng.randint(24, 96), "precision": rng.choice(["f64", "fast"]), "steps": rng.randint(3, 8)}


# ------------------------------------------------------------------ initial data and boundaries
def _extents(case):
    return case["n0"], case["n1"], case["n2"]


def _primitives(case, seed):
    """(eos, mesh, interior primitives [n0, n1, n2, 5] on the GPU, bc) of a
    step, uniform or adjoint case."""
    n = _extents(case)
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    r = torch.rand(8, generator=g, device="cuda", dtype=torch.float64).cpu().tolist()
    mesh = Mesh.new(n, (0.0, 0.0, 0.0), (1.0, 1.0, 1.0), ng=NG)
    axes = [(torch.arange(n[d], device="cuda", dtype=torch.float64) + 0.5) * mesh.dx[d] for d in range(3)]
    x = [axes[0].view(-1, 1, 1), axes[1].view(1, -1, 1), axes[2].view(1, 1, -1)]
    w = torch.zeros(n + (5,), device="cuda", dtype=torch.float64)

    def noise():
        return 2.0 * torch.rand(n, generator=g, device="cuda", dtype=torch.float64) - 1.0

    if case.get("problem") == "waves":
        # Mach-2.5..3 shock into density waves of a stiffened gas, with a weak shear across the channel
        eos = Nasg(1.4, p_inf=0.3)
        k0, k1 = 12.0 + 6.0 * r[0], 2.0 + 2.0 * r[1]
        wave = 0.2 * torch.sin(2 * math.pi * (k0 * x[0] + r[2])) * torch.cos(2 * math.pi * (k1 * x[1] + r[3]))
        post = (x[0] < 0.2 + 0.1 * r[4]).expand(n)
        mach = 2.5 + 0.5 * r[5]
        m2 = mach * mach
        rho2 = 2.4 * m2 / (0.4 * m2 + 2.0)
        c1 = math.sqrt(1.4 * (1.0 + 0.3))
        u2 = mach * c1 * (1.0 - 1.0 / rho2)
        p2 = (1.0 + 0.3) * (1.0 + 2.8 / 2.4 * (m2 - 1.0)) - 0.3
        w[..., 0] = torch.where(post, torch.full(n, rho2, device="cuda", dtype=torch.float64), 1.0 + wave.expand(n))
        w[..., 1] = torch.where(post, u2, 0.0)
        w[..., 2] = 0.05 * torch.sin(2 * math.pi * (x[0] + r[6])).expand(n) * (1 + 0.01 * noise())
        w[..., 4] = torch.where(post, p2, 1.0)
        inflow = (rho2, u2, 0.0, 0.0, p2)
    else:
        # explosion: centre, radius and strength vary; noise on density, small smooth velocities
        eos = Nasg.ideal(1.4)
        r2 = torch.zeros(n, device="cuda", dtype=torch.float64)
        act = [d for d in range(3) if n[d] > 1]
        for d in act:
            r2 = r2 + (x[d] - (0.45 + 0.1 * r[d])) ** 2
        inside = torch.sqrt(r2) < (0.22 + 0.1 * r[3])
        w[..., 0] = torch.where(inside, 1.0, 0.125) * (1.0 + 0.01 * noise())
        w[..., 4] = torch.where(inside, 0.8 + 0.8 * r[4], 0.1) * (1.0 + 0.002 * noise())
        for d in act:
            w[..., 1 + d] = 0.1 * torch.sin(2 * math.pi * (x[act[(d + 1) % len(act)]] + r[5])).expand(n) * (1 + 0.05 * noise())
        inflow = None
    kinds = {"outflow": Bc.Outflow, "periodic": Bc.Periodic, "reflect": Bc.Reflect}
    name = case.get("bc", "outflow")
    if name == "tunnel":
        far = Euler(eos).to_cons(np.array(inflow))
        bc = [[Bc.dirichlet(far), Bc.Outflow], [Bc.Reflect, Bc.Reflect], [Bc.Outflow, Bc.Outflow]]
    else:
        bc = [[kinds[name]] * 2 for _ in range(3)]
    return eos, mesh, w, bc


def _cons(eos, w):
    """Conserved [..., 5] of primitives [..., 5]."""
    rho, p = w[..., 0], w[..., 4]
    ke = 0.5 * rho * (w[..., 1] ** 2 + w[..., 2] ** 2 + w[..., 3] ** 2)
    rhoe = rho * ((p + eos.gamma * eos.p_inf) * (1.0 / rho - eos.b) / (eos.gamma - 1.0) + eos.q)
    return torch.stack([rho, rho * w[..., 1], rho * w[..., 2], rho * w[..., 3], rhoe + ke], dim=-1)


def _initial(case, seed):
    """(eos, mesh, padded AoS conserved state on the GPU, bc)."""
    eos, mesh, w, bc = _primitives(case, seed)
    u = torch.zeros(mesh.padded_shape() + (5,), device="cuda", dtype=torch.float64)
    s = tuple(slice(mesh.g(d), mesh.g(d) + mesh.n[d]) for d in range(3))
    u[s] = _cons(eos, w)
    return eos, mesh, u.view(-1, 5), bc


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


def _riemann(case, seed):
    """The batch of workloads.riemann_batch, built without a loop per instance."""
    ni, nmax = case["ninst"], case["nmax"]
    grids = np.random.default_rng(ni + nmax)  # the set of lines is the case's, their states are the seed's
    n = np.floor(np.exp(grids.uniform(np.log(64), np.log(nmax + 1), ni))).astype(np.int64).clip(64, nmax)
    rng = np.random.default_rng(seed)
    lo, hi = np.array([0.1, -1.0, 0.1] * 2), np.array([2.0, 1.0, 2.0] * 2)
    st = lo + (hi - lo) * rng.random((ni, 6))
    dx = 1.0 / n
    inst = np.repeat(np.arange(ni), n)
    c = np.arange(n.sum()) - np.repeat(np.cumsum(n) - n, n)
    left = (c + 0.5) * dx[inst] < 0.5
    w = np.zeros((len(inst), 5))
    for k, q in enumerate((0, 1, 4)):
        w[:, q] = np.where(left, st[inst, k], st[inst, 3 + k])
    sys_ = Euler(Nasg.ideal(1.4))
    return sys_, n, dx, sys_.to_cons(w)


def _bubble(case, seed):
    """Mach-2 shock and a light bubble of random place and size on the block hierarchy."""
    sys_, cfg, lo, hi, bc, _ = workloads.shock_bubble(dim=case["dim"], base=case["base"], b=16, levels=case["levels"])
    rng = np.random.default_rng(seed)
    centre = 0.5 + 0.04 * rng.uniform(-1.0, 1.0, 3)
    radius, x_shock, tilt = 0.14 + 0.02 * rng.random(), 0.2 + 0.03 * rng.random(), rng.uniform(0.005, 0.02)
    rho2, u2, p2, _ = workloads.rankine_hugoniot(2.0)
    active = range(case["dim"])

    def init(x):
        r2 = sum((x[:, d] - centre[d]) ** 2 for d in active)
        w = np.zeros((x.shape[0], 5))
        w[:, 0] = np.where(r2 < (radius * (1.0 + tilt * np.cos(9.0 * x[:, 1]))) ** 2, 0.138, 1.0)
        w[:, 4] = 1.0
        post = x[:, 0] < x_shock
        w[post, 0], w[post, 1], w[post, 4] = rho2, u2, p2
        return w

    return sys_, cfg, lo, hi, bc, init


def _two_phase(case, seed):
    """Two-phase shock-bubble: a light gas sphere of random place and size in air, Mach-2 shock."""
    n, eps = case["n"], 1e-8
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    r = torch.rand(5, generator=g, device="cuda", dtype=torch.float64).cpu().tolist()
    sys_ = FiveEq((Nasg(1.67), Nasg(1.4)), kapila=True)
    mesh = Mesh.new((n, n, n), (0.0, 0.0, 0.0), (1.0, 1.0, 1.0), ng=NG)
    a = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n
    x = [a.view(-1, 1, 1), a.view(1, -1, 1), a.view(1, 1, -1)]
    rr = sum((x[d] - (0.46 + 0.08 * r[d])) ** 2 for d in range(3))
    inside = torch.sqrt(rr) < 0.14 + 0.02 * r[3]
    rho2, u2, p2, _ = workloads.rankine_hugoniot(2.0)
    post = (x[0] < 0.18 + 0.06 * r[4]).expand(n, n, n)
    al = torch.where(inside, 1.0 - eps, eps).to(torch.float64)
    r1, r2 = al * 0.138, (1.0 - al) * torch.where(post, rho2, 1.0)
    vx = torch.where(post, u2, 0.0).to(torch.float64)
    p = torch.where(post, p2, 1.0).to(torch.float64)
    u = torch.zeros(mesh.padded_shape() + (7,), device="cuda", dtype=torch.float64)
    s = tuple(slice(NG, NG + n) for _ in range(3))
    rho = r1 + r2
    z = torch.zeros_like(rho)
    d = al / (sys_.eos[0].gamma - 1.0) + (1.0 - al) / (sys_.eos[1].gamma - 1.0)
    u[s] = torch.stack([r1, r2, rho * vx, z, z, p * d + 0.5 * rho * vx * vx, al], dim=-1)
    return sys_, mesh, u.view(-1, 7), [[Bc.Outflow, Bc.Outflow] for _ in range(3)]


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind, s = case["kind"], {"case": case}
    prec = PRECISION[case.get("precision", "f64")]
    if kind == "step":
        eos, mesh, u, bc = _initial(case, seed)
        s["mesh"], s["u"] = mesh, u.t().contiguous()  # SoA, as the entry point takes it
        s["out"] = torch.empty_like(s["u"])
        s["args"] = (_c_mesh(mesh), _c_eos(eos), _c_bcs(bc), _abi.EmgOpts(0.5, 1e-3, FluxMode.Weno, 1, prec, 0))
        s["dt"] = 0.1 * min(mesh.dx[:2])
    elif kind == "uniform":
        eos, mesh, u, bc = _initial(case, seed)
        s["mesh"] = mesh
        s["pin"] = _pinned(u), torch.empty(u.shape, dtype=u.dtype, pin_memory=True)
        s["u"], s["out"] = (t.numpy() for t in s["pin"])
        s["solver"] = GpuSolver(Euler(eos), mesh, s["u"], bc=bc, mode=MODE[case["mode"]], precision=prec)
    elif kind == "amr":
        sys_, cfg, lo, hi, bc, init = _bubble(case, seed)
        s["solver"] = GpuAmr(sys_, cfg, lo, hi, bc, init, precision=prec, subcycle=case["subcycle"])
        # host room for every block that the levels could hold, as a program keeps it between outputs
        cap = sum((case["base"] * 2 ** lv) ** case["dim"] for lv in range(case["levels"]))
        s["pin"] = torch.zeros((cap, 16 ** case["dim"], 5), dtype=torch.float64, pin_memory=True)
        s["u"], s["blocks"] = s["pin"].numpy(), np.zeros((cap, 5), dtype=np.int64)
    elif kind == "batch":
        sys_, n, dx, u = _riemann(case, seed)
        s["solver"], s["t"] = GpuBatch1D(sys_, n, dx, u, precision=prec), 0.0
    elif kind == "adjoint":
        eos, mesh, u, bc = _initial(case, seed)
        s["mesh"] = mesh
        s["solver"] = DifferentiableSolver(Euler(eos), mesh, u.cpu().numpy(), bc=bc)
    else:
        sys_, mesh, u, bc = _two_phase(case, seed)
        s["mesh"] = mesh
        s["solver"] = GpuFiveSolver(sys_, mesh, u.cpu().numpy(), bc=bc, precision=prec)
    return s


def run(s):
    case, g = s["case"], s.get("solver")
    kind = case["kind"]
    if kind == "step":
        m, e, b, o = s["args"]
        _abi.check(_abi.lib().emg_uniform_step_noalloc(
            C.byref(m), C.byref(e), b, C.byref(o), s["u"].data_ptr(), s["out"].data_ptr(), s["dt"],
            torch.cuda.current_stream().cuda_stream))
        return s["mesh"].interior(s["out"].t())
    if kind == "uniform":
        g.upload(s["u"])
        g.advance(case["steps"])
        return s["mesh"].interior(g.download(out=s["out"]))
    if kind == "amr":
        for _ in range(case["steps"]):
            if case["subcycle"]:
                g.step_subcycled(g.dt_cfl_subcycled())
            else:
                g.step(g.dt_cfl())
        L, cap = _abi.lib(), len(s["blocks"])
        _abi.check(L.emg_amr_structure(g._h, s["blocks"].ctypes.data_as(C.POINTER(C.c_int64)), cap))
        _abi.check(L.emg_amr_download(g._h, s["u"].ctypes.data_as(C.POINTER(C.c_double)), cap))
        return {"blocks": s["blocks"], "u": s["u"], "count": g.block_count()[0], "t": g.t}
    if kind == "batch":
        s["t"] += case["frame"]
        g.run_to(s["t"])
        return {"u": g.download(), "t": g.status()[0]}
    if kind == "adjoint":
        g.forward(case["steps"])
        J = g.objective(OBJ_PRESSURE if case["objective"] == "pressure" else OBJ_ENERGY, (0.5, 0.0, 0.0), (1.0, 1.0, 1.0))
        ub, wb, gam = g.backward()
        m = s["mesh"]
        return {"J": J, "u": m.interior(g.download()), "ubar": m.interior(ub), "wbar": m.interior(wb), "gamma": gam}
    for _ in range(case["steps"]):
        g.step(g.dt_cfl())
    return s["mesh"].interior(g.download())


# ------------------------------------------------------------------ work and tolerance
# Per cell and stage the state is read and the stage result written, with the
# step's base state in stages 2 and 3: 64 bytes per conserved field and step
# (an adjoint step reads its stage input and cotangents and writes cotangents on
# top of the forward step and its recomputation).
FLOPS_SWEEP = {5: 900, 7: 1300}  # per cell, axis and stage: ten (fourteen) WENO-Z interpolations of ~55, projections, HLLC, limiter


def work(case):
    kind = case["kind"]
    if kind == "amr":
        dim, top = case["dim"], case["base"] * 16 * 2 ** (case["levels"] - 1)
        # finest-level leaves cover the neighbourhood of the shock front and the bubble's surface
        cells, nv = 4.0 * 32 * top ** (dim - 1) + (case["base"] * 16) ** dim, 5
    elif kind == "batch":
        cells, dim, nv = case["ninst"] * (case["nmax"] - 64) / math.log(case["nmax"] / 64), 1, 5
        # every instance takes its own number of steps, proportional to its length
        mean = (case["nmax"] + 64) / 2
        return {"bytes": 64.0 * nv * cells * case["frame"] * mean * 6, "flops": 3.0 * FLOPS_SWEEP[nv] * cells * case["frame"] * mean * 6}
    elif kind == "five":
        cells, dim, nv = case["n"] ** 3, 3, 7
    else:
        n = _extents(case)
        cells, dim, nv = n[0] * n[1] * n[2], sum(1 for m in n if m > 1), 5
    steps = case.get("steps", 1) * (4 if kind == "adjoint" else 1)
    return {"bytes": 64.0 * nv * cells * steps, "flops": 3.0 * dim * FLOPS_SWEEP[nv] * cells * steps}


def tolerance(case):
    """The plain FP64 form rounds every operation as the scheme states it, so
    its results are the same to the last bit; the fast form rounds to about one
    ulp per operation, the mixed form's interpolation is FP32."""
    if case["kind"] == "adjoint":
        return {"rel": 1e-10, "max": 1e-7}
    prec = case["precision"]
    if prec == "f64":
        return "exact"
    if prec == "fast":
        return {"rel": 1e-12, "max": 1e-10}
    return {"rel": 5e-9, "max": 1e-6}


# ------------------------------------------------------------------ the scheme in plain torch, float64
S6 = (75 / 64 - 25 / 384 + 3 / 640, -25 / 384 + 3 / 640, 3 / 640)
A6 = (0.75, -0.15, 1 / 60)


class _Gas:
    def __init__(self, eos, gamma=None):
        self.g = eos.gamma if gamma is None else gamma
        self.pinf, self.b, self.q = eos.p_inf, eos.b, eos.q

    def prim(self, U):
        r = U[0]
        v = [U[k] / r for k in (1, 2, 3)]
        e = U[4] / r - 0.5 * (v[0] ** 2 + v[1] ** 2 + v[2] ** 2)
        return torch.stack([r, *v, (self.g - 1) * (e - self.q) / (1 / r - self.b) - self.g * self.pinf])

    def rhoe(self, W):
        return W[0] * ((W[4] + self.g * self.pinf) * (1 / W[0] - self.b) / (self.g - 1) + self.q)

    def cons(self, W):
        r = W[0]
        return torch.stack([r, r * W[1], r * W[2], r * W[3], self.rhoe(W) + 0.5 * r * (W[1] ** 2 + W[2] ** 2 + W[3] ** 2)])

    def c2(self, W):
        return self.g * (W[4] + self.pinf) / (W[0] * (1 - self.b * W[0]))

    def c(self, W):
        return torch.sqrt(torch.clamp(self.c2(W), min=0.0))

    def ok(self, W):
        return torch.isfinite(W[0]) & torch.isfinite(W[4]) & (W[0] > 0) & (1 / W[0] > self.b) & (W[4] + self.pinf > 0)


def _phys_flux(W, Q, un):
    u = W[un]
    f = [Q[k] * u for k in range(4)] + [(Q[4] + W[4]) * u]
    f[un] = f[un] + W[4]
    return torch.stack(f)


def _weno(a, b, c, d, e):
    q = ((3 * a - 10 * b + 15 * c) / 8, (-b + 6 * c + 3 * d) / 8, (3 * c + 6 * d - e) / 8)
    beta = (13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2,
            13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2,
            13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2)
    tau = torch.abs(beta[0] - beta[2])
    al = [w * (1 + (tau / (x + 1e-40)) ** 2) for w, x in zip((1 / 16, 10 / 16, 5 / 16), beta)]
    return (al[0] * q[0] + al[1] * q[1] + al[2] * q[2]) / (al[0] + al[1] + al[2])


def _hllc(gas, L, R, un):
    cl, cr = gas.c(L), gas.c(R)
    sl, sr = torch.minimum(L[un] - cl, R[un] - cr), torch.maximum(L[un] + cl, R[un] + cr)
    QL, QR = gas.cons(L), gas.cons(R)
    ml, mr = L[0] * (sl - L[un]), R[0] * (sr - R[un])
    ss = (R[4] - L[4] + ml * L[un] - mr * R[un]) / (ml - mr)
    out = None
    for W, Q, s, pick in ((R, QR, sr, ss < 0), (L, QL, sl, ss >= 0)):
        u = W[un]
        fac = W[0] * (s - u) / (s - ss)
        star = [fac, fac * W[1], fac * W[2], fac * W[3], fac * (Q[4] / W[0] + (ss - u) * (ss + W[4] / (W[0] * (s - u))))]
        star[un] = fac * ss
        f = _phys_flux(W, Q, un) + s * (torch.stack(star) - Q)
        out = f if out is None else torch.where(pick, f, out)
    out = torch.where(sr <= 0, _phys_flux(R, QR, un), out)
    return torch.where(sl >= 0, _phys_flux(L, QL, un), out)


def _face_flux(gas, W, un, lam2, mode):
    """Fluxes of the n + 1 faces of lines W[5, ..., n + 10] (five layers on
    each side); lam2 broadcasts over [..., n + 1]."""
    m = W.shape[-1] - 5
    t1, t2 = 1 + un % 3, 1 + (un + 1) % 3
    avg = 0.5 * (W[..., 2:2 + m] + W[..., 3:3 + m])
    rho, c = avg[0], gas.c(avg)
    S = [W[..., s:s + m] for s in range(6)]
    lu, lp, l1 = rho / (2 * c), 1 / (2 * c * c), -1 / (c * c)
    fields = ([-lu * s[un] + lp * s[4] for s in S], [s[0] + l1 * s[4] for s in S], [s[t1] for s in S], [s[t2] for s in S],
              [lu * s[un] + lp * s[4] for s in S])
    sides = []
    for rev in (False, True):
        a = [_weno(*(ch[5:0:-1] if rev else ch[:5])) for ch in fields]
        w = [None] * 5
        w[0], w[un], w[t1], w[t2], w[4] = a[0] + a[1] + a[4], c / rho * (a[4] - a[0]), a[2], a[3], c * c * (a[0] + a[4])
        sides.append(torch.stack(w))
    L, R = sides
    good = gas.ok(L) & gas.ok(R)
    L, R = torch.where(good, L, W[..., 2:2 + m]), torch.where(good, R, W[..., 3:3 + m])
    MF = _hllc(gas, L, R, un)
    n1 = m - 4
    F = S6[0] * MF[..., 2:2 + n1] + S6[1] * (MF[..., 3:3 + n1] + MF[..., 1:1 + n1]) + S6[2] * (MF[..., 4:4 + n1] + MF[..., :n1])
    if mode == "hybrid":
        F = _blend(gas, W, un, F)
    return _limit(gas, W[..., 4:4 + n1], W[..., 5:5 + n1], un, F, lam2)


def _blend(gas, W, un, F):
    """Hybrid switch between the split-form central flux and the shock path."""
    n1 = F.shape[-1]
    rr = torch.zeros_like(F[0])
    for q in (torch.log(W[0]), torch.log(W[4] + gas.pinf)):
        d = torch.abs(q[..., :-4] - 4 * q[..., 1:-3] + 6 * q[..., 2:-2] - 4 * q[..., 3:-1] + q[..., 4:])
        rr = torch.maximum(rr, torch.maximum(d[..., 2:2 + n1], d[..., 3:3 + n1]))
    x = torch.clamp((rr / 1e-3 - 0.5) / 0.5, 0.0, 1.0)
    th = x * x * (3 - 2 * x)
    re, cen = gas.rhoe(W), torch.zeros_like(F)
    for lag in (1, 2, 3):
        for k in range(lag):
            i = 4 - k
            a, b, ea, eb = W[..., i:i + n1], W[..., i + lag:i + lag + n1], re[..., i:i + n1], re[..., i + lag:i + lag + n1]
            u = 0.5 * (a[un] + b[un])
            c = 0.5 * (a[0] + b[0]) * u
            f = [c] + [c * 0.5 * (a[j] + b[j]) for j in (1, 2, 3)]
            f[un] = f[un] + 0.5 * (a[4] + b[4])
            f.append(c * 0.5 * (a[1] * b[1] + a[2] * b[2] + a[3] * b[3]) + u * 0.5 * (ea + eb) + 0.5 * (a[un] * b[4] + b[un] * a[4]))
            cen = cen + 2 * A6[lag - 1] * torch.stack(f)
    return torch.where(th >= 1, F, torch.where(th <= 0, cen, th * F + (1 - th) * cen))


def _limit(gas, A, B, un, F, lam2):
    """Positivity limiter between the cells A and B of each face."""
    UA, UB = gas.cons(A), gas.cons(B)
    FA, FB = _phys_flux(A, UA, un), _phys_flux(B, UB, un)

    def fine(f, ua, ub, fa, fb, l2):
        return gas.ok(gas.prim(ua - l2 * (f - fa))) & gas.ok(gas.prim(ub + l2 * (f - fb)))

    bad = ~(fine(F, UA, UB, FA, FB, lam2) & torch.isfinite(F).all(0)) & (torch.zeros_like(F[0]) + lam2 > 0)
    if not bool(bad.any()):
        return F
    idx = bad.nonzero(as_tuple=True)
    f, ua, ub, fa, fb, a, b = (t[(slice(None),) + idx] for t in (F, UA, UB, FA, FB, A, B))
    l2 = (torch.zeros_like(F[0]) + lam2)[idx]
    alpha = torch.maximum(torch.abs(a[un]) + gas.c(a), torch.abs(b[un]) + gas.c(b))
    low = 0.5 * (fa + fb) - 0.5 * alpha * (ub - ua)
    lo, hi = torch.zeros_like(l2), torch.ones_like(l2)
    for _ in range(30):
        mid = 0.5 * (lo + hi)
        y = fine(torch.where(torch.isfinite(f), mid * f + (1 - mid) * low, low), ua, ub, fa, fb, l2)
        lo, hi = torch.where(y, mid, lo), torch.where(y, hi, mid)
    out = F.clone()
    out[(slice(None),) + idx] = torch.where(torch.isfinite(f), lo * f + (1 - lo) * low, low)
    return out


def _padded(U, ax, bc):
    """Conserved lines U[5, ...] with five boundary layers on both ends of axis ax."""
    n = U.shape[ax]
    parts = []
    for side, b in enumerate(bc):
        if b.kind == Bc.PERIODIC:
            g = U.narrow(ax, n - 5 if side == 0 else 0, 5)
        elif b.kind == Bc.REFLECT:
            g = U.narrow(ax, 0 if side == 0 else n - 5, 5).flip(ax).clone()
            g[ax] = -g[ax]  # momentum 1 + (ax - 1)
        elif b.kind == Bc.DIRICHLET:
            g = torch.tensor(b.state[:5], dtype=U.dtype, device=U.device).view([5] + [1] * (U.dim() - 1))
            g = g.expand_as(U.narrow(ax, 0, 5))
        else:
            g = U.narrow(ax, 0 if side == 0 else n - 1, 1).expand_as(U.narrow(ax, 0, 5))
        parts.append(g)
    return torch.cat([parts[0], U, parts[1]], dim=ax)


def _residual(gas, U, mesh, bc, dt, mode):
    act = [d for d in range(3) if U.shape[1 + d] > 1]
    out = torch.zeros_like(U)
    for d in act:
        P = _padded(U, 1 + d, bc[d])
        lam2 = 2.0 * len(act) * dt / mesh.dx[d]
        if U.requires_grad or U[0].numel() < 1 << 22:
            W = gas.prim(P).movedim(1 + d, -1)
            F = _face_flux(gas, W, 1 + d, lam2, mode)
            out = out - ((F[..., 1:] - F[..., :-1]) / mesh.dx[d]).movedim(-1, 1 + d)
            continue
        lead = 1 if d != 0 else 2  # an axis that is not swept, cut into slabs to bound the memory
        for p, o in zip(P.split(32, dim=lead), out.split(32, dim=lead)):
            F = _face_flux(gas, gas.prim(p).movedim(1 + d, -1), 1 + d, lam2, mode)
            o -= ((F[..., 1:] - F[..., :-1]) / mesh.dx[d]).movedim(-1, 1 + d)
    return out


def _cfl(gas, U, mesh):
    W = gas.prim(U)
    c = gas.c(W)
    return 0.5 / sum((torch.abs(W[1 + d]) + c) / mesh.dx[d] for d in range(3) if U.shape[1 + d] > 1).max()


def _step(gas, U, mesh, bc, dt, mode):
    a = U + dt * _residual(gas, U, mesh, bc, dt, mode)
    b = 0.75 * U + 0.25 * (a + dt * _residual(gas, a, mesh, bc, dt, mode))
    return U / 3 + 2 / 3 * (b + dt * _residual(gas, b, mesh, bc, dt, mode))


def _exact_batch(case, seed):
    """Every instance as one row of a padded array, with its own dx and dt."""
    sys_, n, dx, u = _riemann(case, seed)
    gas, ni, nm = _Gas(sys_.eos), len(n), int(n.max())
    n_, dx = torch.from_numpy(n).cuda(), torch.from_numpy(dx).cuda()
    inst = torch.repeat_interleave(torch.arange(ni, device="cuda"), n_)
    col = torch.arange(len(inst), device="cuda") - torch.repeat_interleave(torch.cumsum(n_, 0) - n_, n_)
    # columns past an instance's end repeat its last cell, as its outflow layers do
    at = torch.minimum(torch.arange(nm, device="cuda").view(1, -1), n_.view(-1, 1) - 1)
    src = (torch.cumsum(n_, 0) - n_).view(-1, 1) + at
    U = torch.from_numpy(u).cuda().t()[:, src]
    pad = torch.clamp(torch.arange(-5, nm + 5, device="cuda").view(1, -1).minimum(n_.view(-1, 1) - 1), min=0)
    pad = pad.unsqueeze(0).expand(5, -1, -1)
    t, end = torch.zeros(ni, device="cuda", dtype=torch.float64), case["frame"]
    while True:
        W = gas.prim(U)
        dt = 0.5 / ((torch.abs(W[1]) + gas.c(W)).amax(1) / dx)
        live = t < end - 1e-10 * end
        if not bool(live.any()):
            break
        dt = torch.where(live, torch.minimum(dt, end - t), 0.0)
        k, h = (dt / dx).view(-1, 1), dt.view(-1, 1)

        def rhs(V):
            F = torch.empty(5, ni, nm + 1, device="cuda", dtype=torch.float64)
            for i in range(0, ni, 512):
                s = slice(i, i + 512)
                F[:, s] = _face_flux(gas, gas.prim(V[:, s].gather(2, pad[:, s])), 1, 2.0 * k[s], "weno")
            d = -(F[..., 1:] - F[..., :-1]) / dx.view(-1, 1)
            return d.gather(2, at.unsqueeze(0).expand(5, -1, -1))

        a = U + h * rhs(U)
        b = 0.75 * U + 0.25 * (a + h * rhs(a))
        U = torch.where(live.view(-1, 1), U / 3 + 2 / 3 * (b + h * rhs(b)), U)
        t = t + dt
    return {"u": U[:, inst, col].t().cpu().numpy(), "t": t.cpu().numpy()}


def _exact_adjoint(case, seed):
    eos, mesh, w, bc = _primitives(case, seed)
    gamma = torch.tensor(eos.gamma, dtype=torch.float64, device="cuda", requires_grad=True)
    gas = _Gas(eos, gamma)
    W0 = w.movedim(-1, 0).clone().requires_grad_(True)
    U0 = gas.cons(W0)
    U0.retain_grad()
    U = U0
    for _ in range(case["steps"]):
        with torch.no_grad():
            dt = _cfl(gas, U, mesh)
        U = _step(gas, U, mesh, bc, dt, "weno")
    box = torch.from_numpy(mesh.centres()[0] >= 0.5).cuda()
    q = gas.prim(U)[4] if case["objective"] == "pressure" else U[4]
    J = (q * box).sum() * math.prod(mesh.dx[d] for d in range(3) if mesh.active(d))
    J.backward()
    at_w = gamma.grad
    at_u = at_w + (U0.grad[4] * W0[4] / (gamma - 1) ** 2).sum().detach()
    aos = lambda t: t.detach().movedim(0, -1).cpu().numpy()  # noqa: E731
    return {"J": float(J), "u": aos(U), "ubar": aos(U0.grad), "wbar": aos(W0.grad),
            "gamma": np.array([float(at_u), float(at_w)])}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("amr", "five"):
        return None
    if kind == "batch":
        return _exact_batch(case, seed)
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    with torch.no_grad():
        eos, mesh, w, bc = _primitives(case, seed)
        gas, U = _Gas(eos), _cons(eos, w).movedim(-1, 0).contiguous()
        mode = case.get("mode", "weno")
        if kind == "step":
            return _step(gas, U, mesh, bc, 0.1 * min(mesh.dx[:2]), mode).movedim(0, -1)
        for _ in range(case["steps"]):
            U = _step(gas, U, mesh, bc, _cfl(gas, U, mesh), mode)
        return U.movedim(0, -1).cpu().numpy()
