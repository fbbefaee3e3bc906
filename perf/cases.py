"""Performance cases of the solver, through its public entry points.

A case is one call sequence a program makes:

  steps    upload a state from pinned host memory, advance it by `steps` RK3
           steps on the device, download it into pinned host memory; with
           `monitor` also what a turbulence run looks at after them (shell
           spectrum, statistics row, residuals, total energy)
  rhs      one right-hand side of device arrays (ns3d_compute_rhs_noalloc)
  adjoint  the gradient of the end-time kinetic energy through `steps` steps

exact() restates the path in 64-bit torch: split, reconstruction, central
viscous terms, Shu-Osher RK3 with the CFL time step, spectrum and statistics.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

import ns3d_cpp_b200 as ns
from ns3d_cpp_b200 import _lib

GAMMA, PR, CFL = 1.4, 0.72, 0.5
TWO_PI = 2.0 * math.pi
SUTHERLAND = 110.4 / 288.15
MDCD_DISS, MDCD_DISP, UD7L_ALPHA = 0.01, 0.0463783, 0.4


def _case(name, call, n, steps, fvs, recon, vis, precision, field, Ma, Re, mach_t=0.0, eps=0.0,
          char=False, monitor=False):
    return {"name": name, "call": call, "nx": n[0], "ny": n[1], "nz": n[2], "steps": steps,
            "fvs": fvs, "recon": recon, "vis": vis, "precision": precision, "field": field,
            "Ma": Ma, "Re": Re, "mach_t": mach_t, "eps": eps, "char": char, "monitor": monitor}


SW, LF = "stagerwarming", "laxfriedrichs"


def listed():
    return [
        # a host program that owns its GPU memory asks for one RHS of a small
        # box at a time: the smallest call, all launches and latency
        _case("rhs_16_fp64", "rhs", (16, 16, 16), 0, SW, "weno5", "c8th", "fp64", "tgv", 0.1, 1600.0),
        # the same call near the largest box it takes, no extent a multiple of
        # 32, FP32-stencil form with an eight-point linear scheme
        _case("rhs_44x36x40_fp32", "rhs", (44, 36, 40), 0, LF, "upwind_7th", "c8th", "fp32acc64",
              "iso", 0.5, 500.0, mach_t=0.3),
        # Taylor-Green vortex at its verification size (the tgv32 workload)
        _case("steps_tgv32_fp64", "steps", (32, 32, 32), 20, SW, "weno5", "c8th", "fp64", "tgv", 0.1,
              1600.0),
        # a coarse parameter study of decaying turbulence in the fast form,
        # with the entropy fix
        _case("steps_iso64_fp32", "steps", (64, 64, 64), 20, SW, "weno5", "c8th", "fp32acc64", "iso",
              0.5, 500.0, mach_t=0.3, eps=1e-3),
        # gradient of the end-time energy (the adjoint workload, fewer steps)
        _case("adjoint_tgv64", "adjoint", (64, 64, 64), 10, SW, "weno5", "c8th", "fp64", "tgv", 0.2,
              400.0, eps=1e-3),
        # the iso128 workload: Lax-Friedrichs + MDCD in FP64 with its monitors
        _case("steps_iso128_mdcd_fp64", "steps", (128, 128, 128), 20, LF, "mdcd", "c8th", "fp64", "iso",
              0.5, 500.0, mach_t=0.3, monitor=True),
        # characteristic-wise reconstruction (the iso128char workload)
        _case("steps_iso128_char_fp64", "steps", (128, 128, 128), 8, SW, "weno5", "c8th", "fp64", "iso",
              0.5, 500.0, mach_t=0.3, char=True),
        # boxes as users choose them, no extent a multiple of 32 or 16
        _case("steps_100x75x90_fp64", "steps", (100, 75, 90), 10, SW, "weno5", "c6th", "fp64", "iso",
              0.5, 500.0, mach_t=0.3),
        _case("steps_150x100x130_fp32", "steps", (150, 100, 130), 20, LF, "ud7l", "c4th", "fp32acc64",
              "iso", 0.5, 500.0, mach_t=0.3),
        # the iso256 workload in both forms: the production size
        _case("steps_iso256_fp32", "steps", (256, 256, 256), 30, SW, "weno5", "c8th", "fp32acc64",
              "iso", 0.5, 1000.0, mach_t=0.5),
        _case("steps_iso256_fp64", "steps", (256, 256, 256), 10, SW, "weno5", "c8th", "fp64", "iso",
              0.5, 1000.0, mach_t=0.5),
        # a large box in the iso512 workload's linear scheme
        _case("steps_iso384_up7_fp32", "steps", (384, 384, 384), 16, SW, "upwind_7th", "c8th",
              "fp32acc64", "iso", 0.5, 2000.0, mach_t=0.4),
    ]


def draw(rng):
    call = rng.choice(["steps"] * 7 + ["rhs"] * 2 + ["adjoint"])
    precision = rng.choice(["fp64", "fp32acc64"])
    recon = rng.choice(["weno5", "weno5", "weno5", "mdcd", "upwind_7th", "ud7l", "linear"])
    char = False
    if call == "rhs":
        lo, hi = 10, 40
    elif call == "adjoint":
        lo, hi, precision = 20, 72, "fp64"
    else:
        char = rng.random() < 0.15
        lo, hi = 20, (140 if char else (220 if precision == "fp64" else 300))
    n0 = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    if rng.random() < 0.5:  # a cube of a round extent, as in the workloads
        q = 32 if n0 >= 96 else (16 if n0 >= 24 else 8)
        n = (max(8, round(n0 / q) * q),) * 3
    else:
        n = tuple(max(8, round(n0 * math.exp(rng.uniform(-0.3, 0.3)))) for _ in range(3))
    while call == "rhs" and n[0] * n[1] * n[2] > 65536:
        n = tuple(max(8, x - 2) for x in n)
    cells = n[0] * n[1] * n[2]
    steps = {"rhs": 0, "adjoint": rng.randint(2, 6)}.get(call)
    if steps is None:
        steps = max(2, min(20, int(6e7 / cells)))
        steps = rng.randint(max(2, steps // 2), steps)
    field = rng.choice(["tgv", "iso"])
    tgv = field == "tgv"
    return {k: v for k, v in _case(
        "", call, n, steps, rng.choice([SW, LF]), recon, rng.choice(["c8th", "c8th", "c6th", "c4th"]),
        precision, field, rng.choice([0.1, 0.2, 0.3]) if tgv else 0.5,
        rng.choice([400.0, 1000.0, 1600.0]), mach_t=0.0 if tgv else rng.choice([0.3, 0.4, 0.5]),
        eps=1e-3 if call == "adjoint" else rng.choice([0.0, 0.0, 1e-3]), char=char,
        monitor=call == "steps" and rng.random() < 0.3).items() if k != "name"}


# ---- inputs -----------------------------------------------------------------

def _solenoidal(n, seed, k0=4.0):
    """Random solenoidal velocity, E(k) ~ k^4 exp(-2 (k/k0)^2), rms component 1."""
    nx, ny, nz = n
    g = torch.Generator(device="cuda").manual_seed(seed)
    kz = torch.fft.fftfreq(nz, 1.0 / nz, dtype=torch.float64, device="cuda").reshape(nz, 1, 1)
    ky = torch.fft.fftfreq(ny, 1.0 / ny, dtype=torch.float64, device="cuda").reshape(1, ny, 1)
    kx = torch.fft.rfftfreq(nx, 1.0 / nx, dtype=torch.float64, device="cuda").reshape(1, 1, -1)
    kk = kx * kx + ky * ky + kz * kz
    amp = torch.sqrt(kk * torch.exp(-2.0 * kk / (k0 * k0)))
    c = [torch.fft.rfftn(torch.randn((nz, ny, nx), dtype=torch.float64, device="cuda", generator=g)) * amp
         for _ in range(3)]
    div = (kx * c[0] + ky * c[1] + kz * c[2]) / torch.where(kk == 0, 1.0, kk)
    u = torch.empty((3, nz, ny, nx), dtype=torch.float64, device="cuda")
    for q, k in enumerate((kx, ky, kz)):
        u[q] = torch.fft.irfftn(c[q] - k * div, s=(nz, ny, nx))
        c[q] = None
    return u / torch.sqrt(torch.mean(u * u))


def _field(case, seed):
    """Initial primitives rho, u, v, w, p of the periodic [0, 2 pi)^3 box."""
    n = (case["nx"], case["ny"], case["nz"])
    W = torch.empty((5, n[2], n[1], n[0]), dtype=torch.float64, device="cuda")
    W[0] = 1.0
    p0 = 1.0 / (GAMMA * case["Ma"] ** 2)
    du = _solenoidal(n, seed)
    if case["field"] == "tgv":  # with a seeded perturbation of amplitude 1e-3
        X, Y, Z = (torch.arange(m, dtype=torch.float64, device="cuda") * (TWO_PI / m) for m in n)
        X, Y, Z = X.reshape(1, 1, -1), Y.reshape(1, -1, 1), Z.reshape(-1, 1, 1)
        W[1] = torch.sin(X) * torch.cos(Y) * torch.cos(Z) + 1e-3 * du[0]
        W[2] = -torch.cos(X) * torch.sin(Y) * torch.cos(Z) + 1e-3 * du[1]
        W[3] = 1e-3 * du[2]
        W[4] = p0 + (torch.cos(2 * X) + torch.cos(2 * Y)) * (torch.cos(2 * Z) + 2.0) / 16.0
    else:  # turbulent Mach number sqrt(<|u|^2>) / c with c = 1 / Ma at T = 1
        W[1:4] = du * (case["mach_t"] / case["Ma"] / math.sqrt(3.0))
        W[4] = p0
    return W


def _params(case):
    p = ns.SolverParams.default().replace(
        gamma=GAMMA, Pr=PR, Ma=case["Ma"], Re=case["Re"], cfl=CFL, dt_fixed=-1.0,
        fvs_type=case["fvs"], recon=case["recon"], vis_scheme=case["vis"], Lx=TWO_PI, Ly=TWO_PI,
        Lz=TWO_PI, precision=case["precision"], char_recon=int(case["char"]),
        sw_entropy_eps=case["eps"], sutherland_s_over_tref=SUTHERLAND, mdcd_diss=MDCD_DISS,
        mdcd_disp=MDCD_DISP, ud7l_alpha=UD7L_ALPHA)
    p.global_nx, p.global_ny, p.global_nz = case["nx"], case["ny"], case["nz"]
    return p.derive()


def prepare(case, seed):
    W = _field(case, seed)
    p = _params(case)
    s = {"case": case, "params": p, "lib": _lib.load()}
    if case["call"] == "rhs":
        s["W"] = W
        s["rhs"] = torch.empty_like(W)
        return s
    s["in"] = torch.empty(W.shape, dtype=torch.float64, pin_memory=True)
    s["in"].copy_(W)
    s["in_np"] = list(s["in"].numpy())
    if case["call"] == "steps":
        s["out"] = torch.empty(W.shape, dtype=torch.float64, pin_memory=True)
        s["out_ptr"] = [ctypes.cast(s["out"][q].data_ptr(), ctypes.POINTER(ctypes.c_double))
                        for q in range(5)]
    s["solver"] = ns.Solver(p)
    return s


# ---- the calls --------------------------------------------------------------

def run(s):
    case, lib = s["case"], s["lib"]
    if case["call"] == "rhs":
        W, rhs = s["W"], s["rhs"]
        st = lib.ns3d_compute_rhs_noalloc(ctypes.byref(s["params"]), *[W[q].data_ptr() for q in range(5)],
                                          rhs.data_ptr(), torch.cuda.current_stream().cuda_stream)
        if st != 0:
            raise ns.NS3DError(st, "ns3d_compute_rhs_noalloc")
        return rhs
    solver = s["solver"]
    solver.upload_primitive(s["in_np"])
    if case["call"] == "adjoint":
        grad, J, dts = solver.adjoint(case["steps"], 5)
        return {"grad": grad, "J": J, "dts": dts}
    solver.step(case["steps"])
    extra = {}
    if case["monitor"]:
        extra = {"total_energy": solver.compute_total_energy(), "residuals": solver.residuals(),
                 "spectrum": solver.compute_energy_spectrum(),
                 "statistics": solver.compute_turbulence_statistics()}
    st = lib.ns3d_download_primitive(solver.ctx, *s["out_ptr"], None, None, ns.solver.LAYOUT["interior"])
    if st != 0:
        raise ns.NS3DError(st, "ns3d_download_primitive")
    return {"state": list(s["out"]), **extra}


def work(case):
    """Compulsory work of one pass. bytes: the five state arrays in and out of
    every call; a stage reads the state and writes the next one, stages 2 and 3
    read the recorded state too (360 B per cell and step with T written). flops: the
    reconstructions (about 70 operations per component, side and direction for
    WENO5, 2 S for an S-point linear scheme), the splits and the viscous terms
    of a right-hand side, the stage update; a reverse step is taken as three
    forward ones."""
    n = case["nx"] * case["ny"] * case["nz"]
    rec = {"weno5": 70.0, "mdcd": 12.0, "linear": 1.0}.get(case["recon"], 16.0)
    rhs = 3.0 * (10.0 * rec + 120.0 + (500.0 if case["char"] else 0.0)) + 400.0
    if case["call"] == "rhs":
        return {"bytes": 80.0 * n, "flops": rhs * n}
    steps = case["steps"] * (4 if case["call"] == "adjoint" else 1)
    return {"bytes": (80.0 + 360.0 * steps) * n, "flops": 3.0 * (rhs + 100.0) * steps * n}


# ---- the same in 64-bit torch -----------------------------------------------

class _Exact:
    """The path on tensors W (5, nz, ny, nx), periodic by torch.roll."""

    def __init__(self, case):
        self.c = case
        n = (case["nx"], case["ny"], case["nz"])
        self.n = n
        self.h = tuple(TWO_PI / m for m in n)
        self.R = 1.0 / (case["Ma"] ** 2 * GAMMA)
        self.Cp = GAMMA / (GAMMA * (GAMMA - 1.0) * case["Ma"] ** 2)
        self.mu0 = 1.0 / case["Re"]
        a, b = UD7L_ALPHA, 1.0 - UD7L_ALPHA
        dp, ds = MDCD_DISP, MDCD_DISS
        self.lin = {
            "linear": [1.0, 0.0],
            "mdcd": [0.5 * (dp + ds), -1.5 * dp - 2.5 * ds - 1 / 12, 7 / 12 + dp + 5 * ds,
                     7 / 12 + dp - 5 * ds, -1.5 * dp + 2.5 * ds - 1 / 12, 0.5 * (dp - ds)],
            "upwind_7th": [-1 / 140, 5 / 84, -101 / 420, 319 / 420, 107 / 210, -19 / 210, 1 / 105, 0.0],
            "ud7l": [-3 / 420 * a - 3 / 840 * b, 25 / 420 * a + 29 / 840 * b,
                     -101 / 420 * a - 139 / 840 * b, 319 / 420 * a + 533 / 840 * b,
                     214 / 420 * a + 533 / 840 * b, -38 / 420 * a - 139 / 840 * b,
                     4 / 420 * a + 29 / 840 * b, -3 / 840 * b]}.get(case["recon"])
        self.S = 6 if self.lin is None else len(self.lin)

    def mu(self, T):
        return self.mu0 * T ** 1.5 * (1.0 + SUTHERLAND) / (T + SUTHERLAND)

    def split(self, W, dim):
        rho, u, v, w, p = W
        vel = (u, v, w)
        k = 0.5 * (u * u + v * v + w * w)
        E = p / (GAMMA - 1.0) + rho * k
        c = torch.sqrt(GAMMA * p / rho)
        un = vel[dim]
        if self.c["fvs"] == SW:
            e = self.c["eps"]
            ls = (un - c, un, un + c)
            ab = [torch.sqrt(x * x + e * e) if e > 0 else x.abs() for x in ls]
            out = []
            for sg in (0.5, -0.5):
                l1, l2, l3 = (0.5 * x + sg * y for x, y in zip(ls, ab))
                s1, s2 = l1 + l3, (l3 - l1) * c
                b = s1 + 2.0 * (GAMMA - 1.0) * l2
                g = rho / (2.0 * GAMMA)
                out.append([g * b] + [g * (b * vel[d] + s2) if d == dim else g * b * vel[d] for d in range(3)]
                           + [g * (s1 * (E + p) / rho + 2.0 * (GAMMA - 1.0) * l2 * k + s2 * un)])
            return out
        am = un.abs() + c
        U = [rho, rho * u, rho * v, rho * w, E]
        F = [x * un for x in U]
        F[1 + dim] = F[1 + dim] + p
        F[4] = F[4] + p * un
        return [[0.5 * (f + sg * am * x) for f, x in zip(F, U)] for sg in (1.0, -1.0)]

    def recon(self, s):
        if self.lin is not None:
            r = self.lin[0] * s[0]
            for c, x in zip(self.lin[1:], s[1:]):
                if c != 0.0:
                    r = r + c * x
            return r
        f0, f1, f2, f3, f4 = s[:5]
        al = []
        for t, e, d in ((f0 - 2 * f1 + f2, f0 - 4 * f1 + 3 * f2, 0.1), (f1 - 2 * f2 + f3, f1 - f3, 0.6),
                        (f2 - 2 * f3 + f4, 3 * f2 - 4 * f3 + f4, 0.3)):
            al.append(d / (1e-6 + 13 / 12 * t * t + 0.25 * e * e) ** 2)
        num = (al[0] * (2 * f0 - 7 * f1 + 11 * f2) + al[1] * (-f1 + 5 * f2 + 2 * f3)
               + al[2] * (2 * f2 + 5 * f3 - f4))
        return num / (6.0 * (al[0] + al[1] + al[2]))

    def faces(self, W, dim):
        """Flux through the face between cells i and i + 1 along dim (x, y, z)."""
        ax, S, mid = 2 - dim, self.S, (self.S - 1) // 2
        at = lambda a, o: torch.roll(a, -o, ax) if o else a  # noqa: E731
        Fp, Fm = self.split(W, dim)
        plus = lambda q: [at(Fp[q], m - mid) for m in range(S)]  # noqa: E731
        minus = lambda q: [at(Fm[q], S - 1 - m - mid) for m in range(S)]  # noqa: E731
        if not self.c["char"]:
            return [self.recon(plus(q)) + self.recon(minus(q)) for q in range(5)]
        l, r = W, torch.stack([at(x, 1) for x in W])
        H = [GAMMA / (GAMMA - 1.0) * x[4] / x[0] + 0.5 * (x[1] ** 2 + x[2] ** 2 + x[3] ** 2) for x in (l, r)]
        sl, sr = torch.sqrt(l[0]), torch.sqrt(r[0])
        avg = lambda a, b: (sl * a + sr * b) / (sl + sr)  # noqa: E731
        u, v, w, h = avg(l[1], r[1]), avg(l[2], r[2]), avg(l[3], r[3]), avg(H[0], H[1])
        nx, ny, nz = (float(dim == d) for d in range(3))
        V = 0.5 * (u * u + v * v + w * w)
        un = (u, v, w)[dim]
        c = torch.sqrt((GAMMA - 1.0) * (h - V))
        t2, t3 = u * nz + v * nx + w * ny, u * ny + v * nz + w * nx
        R = [[1.0, 1.0, 0.0, 0.0, 1.0], [u - c * nx, u, nz, ny, u + c * nx], [v - c * ny, v, nx, nz, v + c * ny],
             [w - c * nz, w, ny, nx, w + c * nz], [h - un * c, V, t2, t3, h + un * c]]
        chi, K = 0.5 / c, (GAMMA - 1.0) / (c * c)
        L = [[0.5 * K * V + chi * un, -chi * nx - 0.5 * K * u, -chi * ny - 0.5 * K * v, -chi * nz - 0.5 * K * w, 0.5 * K],
             [1.0 - K * V, K * u, K * v, K * w, -K], [-t2, nz, nx, ny, 0.0], [-t3, ny, nz, nx, 0.0],
             [0.5 * K * V - chi * un, chi * nx - 0.5 * K * u, chi * ny - 0.5 * K * v, chi * nz - 0.5 * K * w, 0.5 * K]]
        wp, wm = [plus(q) for q in range(5)], [minus(q) for q in range(5)]
        ch = [self.recon([sum(L[q][k] * wp[k][m] for k in range(5)) for m in range(S)])
              + self.recon([sum(L[q][k] * wm[k][m] for k in range(5)) for m in range(S)]) for q in range(5)]
        return [sum(R[q][k] * ch[k] for k in range(5)) for q in range(5)]

    def ddx(self, a, dim):
        ax = 2 - dim
        c = {"c4th": [8 / 12, -1 / 12], "c6th": [45 / 60, -9 / 60, 1 / 60],
             "c8th": [0.8, -0.2, 0.0380952380952381, -0.00357142857142857]}[self.c["vis"]]
        return sum(x * (torch.roll(a, -m, ax) - torch.roll(a, m, ax)) for m, x in enumerate(c, 1)) / self.h[dim]

    def rhs(self, W):
        r = [None] * 5
        for dim in range(3):
            for q, f in enumerate(self.faces(W, dim)):
                d = (torch.roll(f, 1, 2 - dim) - f) / self.h[dim]
                r[q] = d if r[q] is None else r[q] + d
        T = W[4] / (W[0] * self.R)
        mu = self.mu(T)
        g = [[self.ddx(W[1 + q], d) for d in range(3)] for q in range(3)]
        div = g[0][0] + g[1][1] + g[2][2]
        vel = [W[1], W[2], W[3]]
        for d in range(3):
            tau = [mu * (g[q][d] + g[d][q]) - (2 / 3 * mu * div if q == d else 0.0) for q in range(3)]
            e = sum(v * t for v, t in zip(vel, tau)) + mu * self.Cp / PR * self.ddx(T, d)
            for q in range(3):
                r[1 + q] = r[1 + q] + self.ddx(tau[q], d)
            r[4] = r[4] + self.ddx(e, d)
        return torch.stack(r)

    def cons(self, W):
        k = 0.5 * (W[1] ** 2 + W[2] ** 2 + W[3] ** 2)
        return torch.stack([W[0], W[0] * W[1], W[0] * W[2], W[0] * W[3], W[4] / (GAMMA - 1.0) + W[0] * k])

    def prim(self, U):
        u, v, w = U[1] / U[0], U[2] / U[0], U[3] / U[0]
        return torch.stack([U[0], u, v, w, (GAMMA - 1.0) * (U[4] - 0.5 * U[0] * (u * u + v * v + w * w))])

    def dt(self, W):
        a = torch.sqrt(GAMMA * W[4] / W[0])
        return CFL * min(float((h / (W[1 + d].abs() + a)).min()) for d, h in enumerate(self.h))

    def step(self, W, dt):
        U0 = self.cons(W)
        for a, b in ((0.0, 1.0), (0.75, 0.25), (1 / 3, 2 / 3)):
            W = self.prim(a * U0 + b * (self.cons(W) + dt * self.rhs(W)))
        return W

    def spectrum(self, W):
        nx, ny, nz = self.n
        k = [torch.fft.fftfreq(m, 1.0 / m, dtype=torch.float64, device=W.device) for m in (nz, ny, nx)]
        kk = k[0].reshape(-1, 1, 1) ** 2 + k[1].reshape(1, -1, 1) ** 2 + k[2].reshape(1, 1, -1) ** 2
        sh = torch.sqrt(kk).long().reshape(-1)
        E = torch.zeros(2 * nx + 1, dtype=torch.float64, device=W.device)
        for q in (1, 2, 3):
            e = 0.5 * (torch.fft.fftn(W[q]) / W[q].numel()).abs() ** 2
            inside = sh <= 2 * nx
            E.index_add_(0, sh[inside], e.reshape(-1)[inside])
        return E

    def monitors(self, W, W0):
        dV = self.h[0] * self.h[1] * self.h[2]
        q2 = W[1] ** 2 + W[2] ** 2 + W[3] ** 2
        m = lambda a: float(a.mean())  # noqa: E731
        U, U0 = self.cons(W), self.cons(W0)
        res = [math.sqrt(float(((a - b) ** 2).sum()) * self.h[0] ** 3) / float(a.abs().max()) for a, b in zip(U, U0)]
        E = self.spectrum(W)
        T = W[4] / (W[0] * self.R)
        etot = float((0.5 * W[0] * q2).sum()) * dV
        mm, mr, urms, ke = m(self.mu(T)), m(W[0]), math.sqrt(m(q2) / 3.0), 0.5 * m(q2)
        nu = mm / mr
        k = torch.arange(E.numel(), dtype=torch.float64, device=W.device)
        eps = float((2.0 * nu * k * k * E).sum())
        dudx2 = m(self.ddx(W[1], 0) ** 2)
        li = urms / math.sqrt(dudx2)
        st = {"kinetic_energy": ke, "tke": 0.5 * sum(m(W[d] ** 2) - m(W[d]) ** 2 for d in (1, 2, 3)), "u_rms": urms,
              "dissipation": eps, "nu": nu, "mean_mu": mm, "mean_rho": mr,
              "mach_t": math.sqrt(2.0 * ke) / m(torch.sqrt(GAMMA * self.R * T)), "total_energy": etot,
              "taylor": math.sqrt(15.0 * nu * urms ** 2 / eps), "eta": (nu ** 3 / eps) ** 0.25,
              "u_eta": (nu * eps) ** 0.25, "tau_eta": (nu / eps) ** 0.5, "taylor_li": li,
              "re_lambda": urms * li / nu, "dudx2": dudx2}
        return {"total_energy": etot, "residuals": np.array(res), "spectrum": E.cpu().numpy(), "statistics": st}


def exact(case, seed):
    x = _Exact(case)
    W = _field(case, seed)
    if case["call"] == "rhs":
        return x.rhs(W)
    if case["call"] == "steps":
        with torch.no_grad():
            for _ in range(case["steps"]):
                W0, W = W, x.step(W, x.dt(W))
            return {"state": list(W), **(x.monitors(W, W0) if case["monitor"] else {})}
    W = W.requires_grad_(True)
    w, dts = W, []
    for _ in range(case["steps"]):
        dts.append(x.dt(w.detach()))
        U0 = x.cons(w)
        for a, b in ((0.0, 1.0), (0.75, 0.25), (1 / 3, 2 / 3)):
            w = x.prim(a * U0 + b * (x.cons(w) + dts[-1] * checkpoint(x.rhs, w, use_reentrant=False)))
    J = (0.5 * w[0] * (w[1] ** 2 + w[2] ** 2 + w[3] ** 2)).sum() * (x.h[0] * x.h[1] * x.h[2])
    grad, = torch.autograd.grad(J, W)
    return {"grad": grad, "J": float(J.detach()), "dts": np.array(dts)}
