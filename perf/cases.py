"""Workloads of the DUGKS library: what a program that uses it asks of it,
over the range of sizes and options, each through a public entry point.

``listed()`` are the named workloads, ``draw()`` more of the same ranges,
``prepare()`` what a program holds before the call (a solver with its mesh,
DV set, boundary values and start fields), ``run()`` one call, ``work()`` the
bytes and operations it cannot do without, ``exact()`` the same result in
plain torch FP64.

A case's ``kind`` is one of
  step      solver time steps and the cell macros they end in (the shim's
            evolution() loop): mesh cavity | channel | cube | ball, FP64 or FP32C,
            ``steps`` steps per call, ``adaptive`` for the adjustable time step,
            ``K`` internal degrees of freedom (h carried in 3-D), ``nc`` for
            Newton-Cotes nodes (half-range Gauss-Hermite otherwise), ``vmesh`` for
            an unstructured velocity mesh (a DV list)
  adjoint   gradient of wall heat flux and lid shear of a cavity run
  batch     many small cavities stepped through one graph
  restart   a saved state loaded, advanced and saved again
  monitor   cell macros of a caller's device distribution functions
"""
import ctypes
import dataclasses
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "psp-vst_b200", "python"))

from dugks_b200 import case as cs  # noqa: E402
from dugks_b200 import lib as dl  # noqa: E402
from dugks_b200 import meshgen, quadrature  # noqa: E402

# DV updates (cells x DVs x steps) of the largest listed case, which no drawn
# case exceeds
MOST_UPDATES = 110592 * 4096


def listed():
    return [
        # the smallest run anyone makes (the smoke run's size): a call is launches and waits
        dict(name="cavity_smallest", kind="step", mesh="cavity", n=8, n_dv=8, fp32c=False, steps=1),
        # the reference's demo cavity at the benchmark's plain-FP64 size: one evolution() per call, macros read back
        dict(name="cavity_demo", kind="step", mesh="cavity", n=61, n_dv=28, fp32c=False, steps=1),
        # the largest cavity of the batched workload on its own, FP32 storage
        dict(name="cavity_fp32c", kind="step", mesh="cavity", n=256, n_dv=28, fp32c=True, steps=1),
        # a pressure-driven channel with a symmetry side and the adjustable time step, written every few steps; a
        # Newton-Cotes set, whose node at rest is tangential to faces
        dict(name="channel_adaptive", kind="step", mesh="channel", n=47, n_dv=21, nc=True, fp32c=False, steps=4,
             adaptive=True),
        # the headline benchmark: flow past a sphere, far field, 110,592 cells x 16^3 DVs, FP64
        dict(name="ball_far_field", kind="step", mesh="ball", n=24, nr=32, n_dv=16, fp32c=False, steps=1),
        # the lid-driven cube of the mixed-precision configuration (20^3 DVs), FP32 storage
        dict(name="cube_fp32c", kind="step", mesh="cube", n=40, n_dv=20, fp32c=True, steps=1),
        # a gas with internal degrees of freedom in 3-D (h carried), sizes that divide nothing
        dict(name="cube_polyatomic", kind="step", mesh="cube", n=33, n_dv=14, fp32c=False, steps=1, K=2),
        # an unstructured velocity mesh (the reference's VMESH build) around the sphere
        dict(name="ball_velocity_mesh", kind="step", mesh="ball", n=12, nr=14, n_dv=11, fp32c=False, steps=1,
             vmesh=True),
        # sensitivities of a cavity run to its wall temperatures, lid speed and viscosity (32^2 DVs)
        dict(name="adjoint_cavity", kind="adjoint", n=64, n_dv=32, steps=12, snapshots=6),
        # a parameter study: small cavities of several sizes in one graph, FP32 storage
        dict(name="batch_cavities", kind="batch", n=64, n_dv=28, count=12, fp32c=True, steps=2),
        # restart: whole state from host arrays, steps, whole state back to host arrays
        dict(name="restart_cavity", kind="restart", n=61, n_dv=28, fp32c=False, steps=2),
        # a monitor on the caller's own device arrays, between steps
        dict(name="monitor_macros", kind="monitor", n=256, n_dv=28, D=2),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def even(n):
        return n + n % 2

    kind = rng.choice(["step"] * 8 + ["adjoint", "batch", "restart", "monitor"])
    if kind == "adjoint":
        return dict(kind=kind, n=log(12, 96), n_dv=even(rng.randint(8, 32)), steps=rng.randint(4, 12),
                    snapshots=rng.randint(2, 8))
    if kind == "batch":
        return dict(kind=kind, n=log(32, 96), n_dv=even(rng.randint(12, 28)), count=rng.randint(4, 12),
                    fp32c=rng.random() < 0.7, steps=rng.randint(1, 4))
    if kind == "restart":
        return dict(kind=kind, n=log(12, 80), n_dv=even(rng.randint(8, 32)), fp32c=rng.random() < 0.3,
                    steps=rng.randint(1, 4))
    if kind == "monitor":
        D = rng.choice([2, 3])
        return dict(kind=kind, n=log(32, 300) if D == 2 else log(12, 40), D=D,
                    n_dv=even(rng.randint(8, 32) if D == 2 else rng.randint(6, 14)))
    while True:
        mesh = rng.choice(["cavity", "cavity", "channel", "ball", "cube"])
        d3 = mesh in ("ball", "cube")
        c = dict(kind=kind, mesh=mesh, fp32c=rng.random() < 0.4, steps=rng.choice([1, 1, 2, 5]))
        c["n"] = even(log(3, 23)) if mesh == "ball" else log(6, 48) if mesh == "cube" else log(8, 256)
        c["n_dv"] = even(rng.randint(6, 20) if d3 else log(6, 40))
        if rng.random() < 0.25:
            c["nc"], c["n_dv"] = True, 4 * max(2, c["n_dv"] // 4) + 1
        if mesh == "ball":
            c["nr"] = log(4, 32)
        if mesh == "channel" or rng.random() < 0.15:
            c["adaptive"] = True
        if d3 and rng.random() < 0.3:
            c["K"] = 2
        if not c.get("adaptive") and mesh != "channel" and rng.random() < 0.15:
            c.pop("nc", None)
            c["vmesh"], c["n_dv"] = True, rng.randint(6, 12)
        u = cells_of(c) * c["n_dv"] ** dims_of(c) * c["steps"] * (2 if c.get("vmesh") else 1)
        if u * (1 if d3 and not c.get("K") else 2) <= MOST_UPDATES // 2:
            return c


def dims_of(case):
    return case["D"] if "D" in case else 3 if case.get("mesh") in ("ball", "cube") else 2


def cells_of(case):
    n = case["n"]
    if case["kind"] == "monitor":
        return n ** case["D"]
    mesh = case.get("mesh", "cavity")
    return {"cavity": n * n, "channel": 2 * n * n, "cube": n ** 3, "ball": 6 * n * n * case.get("nr", 0)}[mesh]


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=8)
def base_case(mesh, n, nr, n_dv, nc, vmesh):
    """The mesh and DV set of a case, as a program reads them once."""
    sets, n_dv = n_dv, 8 if nc or vmesh else n_dv
    if mesh == "cavity":
        c = cs.cavity_case(n, n_dv, kn=0.1)
    elif mesh == "channel":
        # pressure patches start at density one, so this gas is scaled to it at the same Knudsen number
        p = cs.R_DEMO * 273.0
        c = cs.channel_case(2 * n, n, n_dv, kn=0.1, sides={
            "inlet": {"kind": "pressureIn", "p": 1.2 * p, "T": 273.0}, "outlet": {"kind": "pressureOut", "p": p},
            "bottom": {"kind": "maxwellWall"}, "top": {"kind": "symmetryPlane"}})
        c.gas["muRef"] /= float(c.rho0[0])
        c.rho0 = np.ones(c.n_cells)
    elif mesh == "cube":
        c = cs.cube_case(n, n_dv, kn=0.1)
    else:
        c = cs.ball_case(n, nr, 1.12, n_dv, kn=0.1, mach=0.5)
    v = 4.0 * math.sqrt(2.0 * c.gas["R"] * 273.0)
    if nc:
        c.xis, c.weights = quadrature.newton_cotes(v, sets)
        c.xi_max = v
    if vmesh:
        c.use_velocity_mesh(meshgen.velocity_box(sets, v, c.D, jitter=0.2))
    c.dt = cs.cfl_dt(c, 0.5)
    return c


def user_case(case, seed, n=None, lid=None):
    """One user's case: wall temperatures about 273 K, and start fields with
    smooth variations of a developing flow (all seeded)."""
    b = base_case(case.get("mesh", "cavity"), n or case["n"], case.get("nr", 0), case["n_dv"],
                  bool(case.get("nc")), bool(case.get("vmesh")))
    rng = np.random.default_rng(seed)
    fl = dict(b.flat)
    wall = np.repeat(fl["patch_type"] == 1, np.diff(fl["patch_start"]))
    fl["T_b"] = np.where(wall, fl["T_b"] + rng.normal(0.0, 5.0, len(wall)), fl["T_b"])
    if lid is not None:
        U_b = np.array(fl["U_b"])
        U_b[:fl["patch_start"][1], 0] = lid
        fl["U_b"] = U_b
    x = fl["C"] / np.abs(fl["C"]).max()

    def wave():
        k, p = rng.integers(1, 4, 3), rng.uniform(0, 2 * np.pi)
        return np.sin(np.pi * (x @ k) + p)

    U0 = b.U0 + 15.0 * np.stack([wave(), wave(), wave() if b.D == 3 else 0 * x[:, 0]], axis=1)
    gas = dict(b.gas, K=case.get("K", 0))
    return dataclasses.replace(b, flat=fl, gas=gas, rho0=b.rho0 * (1 + 0.04 * wave()), U0=U0,
                               T0=b.T0 * (1 + 0.02 * wave()))


def batch_cases(case, seed):
    """Cavities of several sides, lid speeds uniform in [10, 100] m/s."""
    rng = np.random.default_rng(seed)
    sides = [max(8, int(case["n"] * f)) for f in (0.5, 0.75, 1.0, 1.5)]
    return [user_case(case, seed * 1000 + i, n=sides[i % 4], lid=rng.uniform(10.0, 100.0))
            for i in range(case["count"])]


def states(case, seed):
    """g~, h~ of a saved run, DV-major [n_dv][cells]: the Maxwellian of the
    start fields with the tails a flow has."""
    c = user_case(case, seed)
    xi, _ = c.dv_set()
    rng = np.random.default_rng(seed + 1)
    RT = c.gas["R"] * c.T0
    c2 = ((xi[:, None, 0] - c.U0[:, 0]) ** 2 + (xi[:, None, 1] - c.U0[:, 1]) ** 2 +
          (xi[:, None, 2] - c.U0[:, 2]) ** 2) / RT
    g = c.rho0 / (2 * np.pi * RT) ** (c.D / 2) * np.exp(-0.5 * c2)
    g *= 1 + 0.02 * np.tanh(rng.normal(size=(len(xi), 1))) * np.sin(3 * c.flat["C"][:, 0] + rng.uniform(0, 6))
    return c, g, (c.gas["K"] + 3 - c.D) * RT * g


def monitor_arrays(case, seed):
    """The caller's own arrays: xi, w, g, h on the device and its gas."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    D, n = case["D"], cells_of(case)
    b = base_case("cavity" if D == 2 else "cube", 4, 0, case["n_dv"], False, False)
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    xi, w = (torch.as_tensor(a, device=dev).contiguous() for a in b.dv_set())
    RT = b.gas["R"] * 273.0 * (1 + 0.05 * torch.rand(n, generator=gen, device=dev, dtype=torch.float64))
    U = 30.0 * torch.randn(D, n, generator=gen, device=dev, dtype=torch.float64)
    c2 = sum((xi[:, k, None] - U[k]) ** 2 for k in range(D)) / RT
    g = float(b.rho0[0]) / (2 * math.pi * RT) ** (D / 2) * torch.exp(-0.5 * c2)
    g = g * (1 + 0.01 * torch.rand(len(w), 1, generator=gen, device=dev, dtype=torch.float64))
    gas = dict(b.gas)
    return b, xi, w, g.contiguous(), ((gas["K"] + 3 - D) * RT * g).contiguous(), gas


class State:
    pass


def prepare(case, seed):
    s = State()
    s.case, s.kind = case, case["kind"]
    prec = dl.FP32C if case.get("fp32c") else dl.FP64
    if s.kind == "batch":
        cases = batch_cases(case, seed)
        s.solvers = [dl.Solver(c, precision=prec) for c in cases]
        s.batch = dl.Batch(s.solvers, [c.dt for c in cases])
    elif s.kind == "monitor":
        s.base, s.xi, s.w, s.g, s.h, g = monitor_arrays(case, seed)
        s.gas = dl.Gas(g["R"], g["omega"], g["Tref"], g["muRef"], g["Pr"], int(g["K"]))
        s.lib, s.msg = dl.load(), ctypes.create_string_buffer(256)
        n = s.g.shape[1]
        s.out = {"rho": torch.empty(n, dtype=torch.float64, device="cuda"),
                 "U": torch.empty(n, 3, dtype=torch.float64, device="cuda"),
                 "T": torch.empty(n, dtype=torch.float64, device="cuda"),
                 "q": torch.empty(n, 3, dtype=torch.float64, device="cuda")}
    elif s.kind == "restart":
        c, s.g, s.h = states(case, seed)
        s.solver = dl.Solver(c, precision=prec)
    else:
        c = user_case(case, seed)
        s.solver = dl.Solver(c, precision=prec)
        if s.kind == "adjoint":
            s.ew, s.mw = objective_of(c)
    return s


def objective_of(c):
    """Wall heat flux on every wall face and x-momentum flux on the lid."""
    nb = c.flat["n_boundary"]
    mw = np.zeros((nb, 3))
    mw[:c.flat["patch_start"][1], 0] = 1.0
    return np.ones(nb), mw


def run(s):
    case = s.case
    if s.kind == "batch":
        s.batch.step(case["steps"])
        return [x.macros() for x in s.solvers]
    if s.kind == "monitor":
        o = s.out
        st = s.lib.dugks_cell_macros_noalloc(
            case["D"], s.w.numel(), s.xi.data_ptr(), s.w.data_ptr(), s.g.shape[1], s.g.data_ptr(), s.h.data_ptr(),
            ctypes.byref(s.gas), s.base.dt, o["rho"].data_ptr(), o["U"].data_ptr(), o["T"].data_ptr(),
            o["q"].data_ptr(), torch.cuda.current_stream().cuda_stream, s.msg, len(s.msg))
        if st != 0:
            raise RuntimeError(s.msg.value.decode())
        return o
    sv = s.solver
    dt = sv.case.dt
    if s.kind == "adjoint":
        r = sv.adjoint(case["steps"], dt, s.ew, s.mw, window_start=case["steps"] // 4,
                       max_snapshots=case["snapshots"])
        return {k: r[k] for k in ("J", "dT_b", "dU_b", "dmu")}
    if s.kind == "restart":
        sv.set_state(s.g, s.h, dt)
        sv.step(case["steps"], dt)
        g, h = sv.state()
        return {"g": g, "h": h, "macros": sv.macros()}
    if case.get("adaptive"):
        last, hist = sv.step_adaptive(case["steps"], dt, 0.8)
        return dict(sv.macros(), dt=hist)
    if case["steps"] == 1:
        sv.evolution(dt)
    else:
        sv.step(case["steps"], dt)
    return sv.macros()


# ---------------------------------------------------------------------------
# what a call cannot do without
# ---------------------------------------------------------------------------
# FP64 operations per (cell, DV) and step: the cell's relaxation (14) and
# update (4), its gradient (about 7 per neighbour and dimension pair), per face
# the reconstruction (2 D), relaxation (14), flux (2 D) and the moments (8),
# the cell's moments (8); faces per cell: D
def work(case):
    D = dims_of(case)
    cells, nv = cells_of(case), case["n_dv"] ** D
    real = 4 if case.get("fp32c") else 8
    fields = 2 if D == 2 or case.get("K") or case["kind"] == "monitor" else 1   # 3-D, K = 0: h is identically zero
    if case["kind"] == "monitor":
        return {"bytes": cells * nv * 2 * 8 + cells * 64, "flops": cells * nv * 24}
    per = fields * (26 + 2 * D * (1 + 2 * D) + D * (4 * D + 14) + 8 * (1 + D))
    if case["kind"] == "batch":
        sides = [max(8, int(case["n"] * f)) for f in (0.5, 0.75, 1.0, 1.5)]
        cells = sum(sides[i % 4] ** 2 for i in range(case["count"]))
    updates = cells * nv * case["steps"]
    if case["kind"] == "adjoint":
        # a forward step and a reversed one, which reads the state and its adjoint and writes the latter
        return {"bytes": updates * fields * 8 * (3 + 4), "flops": updates * per * 4}
    # each step reads the state for the face values, again for the update, and writes it
    b = updates * fields * real * 3 + cells * 64
    if case["kind"] == "restart":
        b += 2 * cells * nv * 2 * 8
    return {"bytes": b, "flops": updates * per}


# ---------------------------------------------------------------------------
# the same results in plain torch, 64 bits
# ---------------------------------------------------------------------------
class Exact:
    """One DUGKS run (fvDVM::evolution) over whole arrays [dv][entity]."""

    def __init__(self, c, whole=False):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.c, self.D, fl = c, c.D, c.flat
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=self.dev)  # noqa: E731
        self.g = dict(c.gas)
        self.mu = torch.tensor(c.gas["muRef"], dtype=torch.float64, device=self.dev)
        xi, w = c.dv_set()
        self.xi, self.w = t(xi), t(w)
        self.nIF, self.nBF, self.nC = fl["n_internal"], fl["n_boundary"], c.n_cells
        own = t(fl["owner"])
        self.own, self.nei, self.bown = own[:self.nIF], t(fl["neighbour"]), own[self.nIF:]
        self.allown = own
        self.S, self.V = t(fl["Sf"]), t(fl["V"])
        C, Cf = t(fl["C"]), t(fl["Cf"])
        self.dO = Cf - C[own]
        self.dN = Cf[:self.nIF] - C[self.nei]
        self.lsP, self.lsN = self.least_squares(C, Cf)
        d = C[self.nei] - C[self.own]
        self.dc = 1 / d.norm(dim=1)
        so = (self.S[:self.nIF] * self.dO[:self.nIF]).sum(1).abs()
        sn = (self.S[:self.nIF] * self.dN).sum(1).abs()
        self.lin = (sn / (so + sn))[:, None]
        counts = np.diff(fl["patch_start"])
        self.ptype = t(np.repeat(fl["patch_type"], counts).astype(np.int64))
        first = np.repeat(fl["patch_start"][:-1], counts)
        self.first = t(first.astype(np.int64))
        self.local = t((np.arange(self.nBF) - first).astype(np.int64))
        self.rho_b, self.U_b, self.T_b, self.p_b = (t(fl[k]).clone() for k in ("rho_b", "U_b", "T_b", "p_b"))
        self.K3D = c.gas["K"] + 3 - self.D
        nv = len(w)
        size = nv if whole else max(1, min(nv, 24_000_000 // max(1, len(own))))
        self.slices = [slice(a, min(nv, a + size)) for a in range(0, nv, size)]
        self.mirror = None
        if bool(((self.ptype == 5) | (self.ptype == 6)).any()):
            n, D = len(c.xis), self.D
            i = torch.arange(nv, device=self.dev)
            k = [i % n, (i // n) % n, i // (n * n) if D == 3 else 0 * i]
            self.mirror = [i + (n - 1 - 2 * k[a]) * n ** a for a in range(D)]
            self.slices = [slice(0, nv)]

    def least_squares(self, C, Cf):
        D, nIF = self.D, self.nIF
        mag = self.S.norm(dim=1)
        d = (C[self.nei] - C[self.own])[:, :D]
        c = mag[:nIF] / (C[self.nei] - C[self.own]).square().sum(1)
        so = (self.S[:nIF] * (Cf[:nIF] - C[self.own])).sum(1).abs()
        sn = (self.S[:nIF] * (C[self.nei] - Cf[:nIF])).sum(1).abs()
        w = sn / (so + sn)
        fo, fn = (1 - w) * c, w * c
        nrm = self.S[nIF:] / mag[nIF:, None]
        bd3 = nrm * (nrm * (Cf[nIF:] - C[self.bown])).sum(1, keepdim=True)
        bd = bd3[:, :D]
        fb = mag[nIF:] / bd3.square().sum(1)
        dd = torch.zeros(self.nC, D, D, dtype=torch.float64, device=self.dev)
        sq = d[:, :, None] * d[:, None, :]
        dd.index_add_(0, self.own, fo[:, None, None] * sq)
        dd.index_add_(0, self.nei, fn[:, None, None] * sq)
        dd.index_add_(0, self.bown, fb[:, None, None] * bd[:, :, None] * bd[:, None, :])
        inv = torch.linalg.inv(dd)
        return fo[:, None] * torch.einsum("nij,nj->ni", inv[self.own], d), \
            -fn[:, None] * torch.einsum("nij,nj->ni", inv[self.nei], d)

    def tau(self, rho, T):
        return self.mu * (T / self.g["Tref"]) ** self.g["omega"] / rho / T / self.g["R"]

    def maxwell(self, xi, rho, U, T):
        RT = self.g["R"] * T
        c2 = sum((xi[:, k, None] - U[:, k]) ** 2 for k in range(self.D))
        return rho / (2 * math.pi * RT) ** (self.D / 2) * torch.exp(-0.5 * c2 / RT)

    def relax(self, sl, g, h, m, r, RTh=None):
        """(1 - r) f + r f^S (fvDVM.C:648-683, :1362-1457)"""
        rho, U, T, q = m
        xi, RT = self.xi[sl], self.g["R"] * T
        cs2 = sum((xi[:, k, None] - U[:, k]) ** 2 for k in range(self.D)) / RT
        s = sum((xi[:, k, None] - U[:, k]) * q[:, k] for k in range(self.D)) * (1 - self.g["Pr"]) / (5 * rho * RT * RT)
        E = self.maxwell(xi, rho, U, T)
        gS = E * (1 + s * (cs2 - self.D - 2))
        hS = E * (RT if RTh is None else RTh) * (self.K3D + s * ((cs2 - self.D) * self.K3D - 2 * self.g["K"]))
        return (1 - r) * g + r * gS, (1 - r) * h + r * hS

    def moments(self, sl, g, h):
        xi, w = self.xi[sl], self.w[sl, None]
        x2 = xi.square().sum(1)[:, None]
        u = w * (x2 * g + h)
        a = w * g
        M = lambda f, k: (f * xi[:, k, None]).sum(0)  # noqa: E731
        D = self.D
        return torch.stack([a.sum(0), u.sum(0)] + [M(a, k) for k in range(D)] + [M(u, k) for k in range(D)] +
                           [(a * (xi[:, i] * xi[:, j])[:, None]).sum(0) for i in range(D) for j in range(i, D)])

    def macros(self, s, dtPr):
        """rho, U, T, q, tau from raw moments, q reduced by 2 tau / (2 tau + dt Pr)"""
        D, K, R = self.D, self.g["K"], self.g["R"]
        rho = s[0]
        U = torch.stack([s[2 + k] / rho if k < D else 0 * rho for k in range(3)], 1)
        u2 = U.square().sum(1)
        T = (0.5 * s[1] - 0.5 * rho * u2) / ((K + 3) / 2 * R * rho)
        tau = self.tau(rho, T)
        M2, at = {}, 2 + 2 * D
        for i in range(D):
            for j in range(i, D):
                M2[i, j] = M2[j, i] = s[at]
                at += 1
        q = torch.stack([0.5 * (s[2 + D + i] - 2 * sum(M2[i, j] * U[:, j] for j in range(D)) - U[:, i] * s[1] +
                                2 * rho * u2 * U[:, i]) if i < D else 0 * rho for i in range(3)], 1)
        return rho, U, T, q * (2 * tau / (2 * tau + dtPr))[:, None], tau

    @staticmethod
    def dot(xi, S):
        """xi . S term by term as the reference rounds it: its sign picks the upwind side"""
        return (xi[:, 0, None] * S[:, 0] + xi[:, 1, None] * S[:, 1]) + xi[:, 2, None] * S[:, 2]

    def add(self, base, index, src):
        return base.index_add(1, index, src)

    def face_values(self, sl, g, h, m, r, dt):
        """half-step face values of every face before the relaxation; incoming wall ones are zero"""
        gb, hb = self.relax(sl, g, h, m[:4], r)
        xi, D, n = self.xi[sl], self.D, self.nIF
        xs = self.dot(xi, self.S)
        out = []
        for f in (gb, hb):
            d = f[:, self.nei] - f[:, self.own]
            grad = []
            for k in range(D):
                z = torch.zeros_like(f)
                z = self.add(z, self.own, d * self.lsP[:, k])
                grad.append(self.add(z, self.nei, -d * self.lsN[:, k]))

            def rec(cell, dist):
                v = f[:, cell]
                for k in range(D):
                    v = v + grad[k][:, cell] * (dist[:, k] - 0.5 * dt * xi[:, k, None])
                return v

            a, b = rec(self.own, self.dO[:n]), rec(self.nei, self.dN)
            x = xs[:, :n]
            inner = torch.where(x >= 1e-300, a, torch.where(x < -1e-300, b, 0.5 * (a + b)))
            out.append((inner, rec(self.bown, self.dO[n:]), f[:, self.bown]))
        return xs, gb, hb, out

    def boundary(self, sl, xs, vals, m, rho_w, mirror):
        """boundary face values with the incoming DFs (fvDVM.C:866-1098)"""
        xi, pt = self.xi[sl], self.ptype
        xb = xs[:, self.nIF:]
        (g, h), (gc, hc) = (vals[0][1], vals[1][1]), (vals[0][2], vals[1][2])
        U = torch.where(((pt == 1) | (pt == 4))[:, None], self.U_b, m[1][self.bown])
        T = torch.where((pt == 3) | (pt >= 5) & (pt <= 6), torch.full_like(self.T_b, 273.0), self.T_b)
        rho = torch.where(pt == 1, rho_w, self.rho_b)
        gi = self.maxwell(xi, rho, U, T)
        hi = gi * self.g["R"] * T * self.K3D
        inc = xb <= 0
        if mirror:
            # symmetry: the incoming DVs of the patch's first face take their mirror's face value
            S0 = self.S[self.nIF + self.first]
            sym = (pt == 5) | (pt == 6)
            axis = S0.abs()[:, :self.D].argmax(1)
            i0 = self.dot(xi, S0) <= 0
            gm = torch.stack([g[self.mirror[a]] for a in range(self.D)])
            hm = torch.stack([h[self.mirror[a]] for a in range(self.D)])
            pick = axis[None, None, :].expand(1, len(xi), -1)
            gs, hs = gm.gather(0, pick)[0], hm.gather(0, pick)[0]
            g, h = torch.where(inc & ~sym, gi, g), torch.where(inc & ~sym, hi, h)
            g, h = torch.where(i0 & sym, gs, g), torch.where(i0 & sym, hs, h)
        else:
            g, h = torch.where(inc, gi, g), torch.where(inc, hi, h)
        z = pt == 3
        return torch.where(z, gc, g), torch.where(z, hc, h), inc

    def step(self, g, h, m, dt, flux_sum=None):
        """one step: new g~, h~, macros; the largest Courant number per unit time step"""
        n, R = self.nIF, self.g["R"]
        rc = 1.5 * dt / (2 * m[4] + dt)
        wall = self.ptype == 1
        kept, out_w, in_w, sums = [], 0, 0, 0
        unit = torch.ones_like(self.rho_b)
        for sl in self.slices:
            xs, gb, hb, vals = self.face_values(sl, g[sl], h[sl], m, rc, dt)
            xb, w = xs[:, n:], self.w[sl, None]
            out_w = out_w + torch.where(xb > 0, w * xb * vals[0][1], 0 * xb).sum(0)
            in_w = in_w + torch.where(xb < 0, -w * xb * self.maxwell(self.xi[sl], unit, self.U_b, self.T_b),
                                      0 * xb).sum(0)
            kept.append((sl, xs, gb, hb, vals))
            if len(self.slices) > 1:
                kept[-1] = (sl, xs, None, None, vals)
        rho_w = out_w / in_w.abs()
        for k, (sl, xs, gb, hb, vals) in enumerate(kept):
            gB, hB, inc = self.boundary(sl, xs, vals, m, rho_w, self.mirror)
            gf, hf = torch.cat([vals[0][0], gB], 1), torch.cat([vals[1][0], hB], 1)
            sums = sums + self.moments(sl, gf, hf)
            kept[k] = (sl, xs, gb, hb, gf, hf, inc)
        f = self.macros(sums, 0.5 * dt * self.g["Pr"])
        rf = 0.5 * dt / (2 * f[4] + 0.5 * dt)
        RTh = torch.cat([R * f[2][:n], R * f[2][self.local]])
        gn, hn, csum = [], [], 0
        for sl, xs, gb, hb, gf, hf, inc in kept:
            if gb is None:
                gb, hb = self.relax(sl, g[sl], h[sl], m[:4], rc)
            ga, ha = self.relax(sl, gf, hf, f[:4], rf, RTh)
            no = torch.cat([torch.zeros(len(inc), n, dtype=torch.bool, device=self.dev), inc], 1)
            ga, ha = torch.where(no, gf, ga), torch.where(no, hf, ha)
            if flux_sum is not None:
                flux_sum(self, sl, xs[:, n:], ga[:, n:], ha[:, n:])
            new = []
            for old, bar, fl in ((g[sl], gb, xs * ga), (h[sl], hb, xs * ha)):
                d = self.add(torch.zeros_like(old), self.allown, fl)
                d = self.add(d, self.nei, -fl[:, :n])
                new.append(-old / 3 + 4 / 3 * bar - dt / self.V * d)
            csum = csum + self.moments(sl, *new)
            gn.append(new[0])
            hn.append(new[1])
        m = self.macros(csum, dt * self.g["Pr"])
        self.pressures(m)
        co = (self.dc * (f[1][:n].norm(dim=1) + math.sqrt(self.D) * self.c.xi_max)).max()
        return torch.cat(gn), torch.cat(hn), m, co

    def pressures(self, m):
        """pressureIn / pressureOut patch values after the step (fvDVM.C:1745-1821)"""
        pin, pout = self.ptype == 7, self.ptype == 8
        if not bool((pin | pout).any()):
            return
        R, K = self.g["R"], self.g["K"]
        rho, T = m[0][self.bown], m[2][self.bown]
        a2 = R * T * (K + 5) / (K + 3)
        self.rho_b = torch.where(pin, self.p_b / R / self.T_b,
                                 torch.where(pout, rho + (self.p_b - rho * R * T) / a2, self.rho_b))
        self.T_b = torch.where(pout, self.p_b / (R * rho), self.T_b)

    def start(self):
        c = self.c
        t = lambda a: torch.as_tensor(a, device=self.dev, dtype=torch.float64)  # noqa: E731
        rho, U, T = t(c.rho0), t(c.U0), t(c.T0)
        g = torch.cat([self.maxwell(self.xi[sl], rho, U, T) for sl in self.slices])
        return g, g * (self.K3D * self.g["R"] * T), (rho, U, T, 0 * U, self.tau(rho, T))


def told(m):
    return {k: m[i].detach().cpu().numpy() for i, k in enumerate(("rho", "U", "T", "q"))}


def exact_step(case, c):
    e = Exact(c)
    g, h, m = e.start()
    dt, hist = c.dt, []
    Uf = e.lin * (m[1][e.own] - m[1][e.nei]) + m[1][e.nei]
    co = (e.dc * (Uf.norm(dim=1) + math.sqrt(e.D) * c.xi_max)).max()
    for _ in range(case["steps"]):
        if case.get("adaptive"):
            F = 0.8 / (float(co) * dt + 1e-15)
            dt = dt * min(min(F, 1 + 0.1 * F), 1.2)
            hist.append(dt)
        g, h, m, co = e.step(g, h, m, dt)
    return dict(told(m), dt=np.array(hist)) if case.get("adaptive") else told(m)


def exact_adjoint(case, c):
    e = Exact(c, whole=True)
    ew, mw = (torch.as_tensor(a, device=e.dev) for a in objective_of(c))
    steps, first, J = case["steps"], case["steps"] // 4, [0.0]
    for p in (e.T_b, e.U_b, e.mu):
        p.requires_grad_(True)
    g, h, m = e.start()
    m = tuple(x.detach() for x in m)

    def objective(e, sl, xb, ga, ha):
        xi, w = e.xi[sl], e.w[sl, None]
        J[0] = J[0] + (w * xb * (ew * 0.5 * (xi.square().sum(1)[:, None] * ga + ha) +
                                 (xi @ mw.T) * ga)).sum() / (steps - first)

    for n in range(steps):
        g, h, m, _ = e.step(g, h, m, c.dt, objective if n >= first else None)
    dT, dU, dmu = torch.autograd.grad(J[0], (e.T_b, e.U_b, e.mu))
    return {"J": float(J[0].detach()), "dT_b": dT.cpu().numpy(), "dU_b": dU.cpu().numpy(), "dmu": float(dmu)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "monitor":
        b, xi, w, g, h, gas = monitor_arrays(case, seed)
        e = Exact(b)
        s = sum(e.moments(slice(a, a + 64), g[a:a + 64], h[a:a + 64]) for a in range(0, len(w), 64))
        return told(e.macros(s, b.dt * gas["Pr"]))
    if kind == "batch":
        return [exact_step(case, c) for c in batch_cases(case, seed)]
    if kind == "restart":
        c, g, h = states(case, seed)
        e = Exact(c)
        g, h = (torch.as_tensor(a, device=e.dev) for a in (g, h))
        s = sum(e.moments(sl, g[sl], h[sl]) for sl in e.slices)
        m = e.macros(s, c.dt * c.gas["Pr"])
        for _ in range(case["steps"]):
            g, h, m, _ = e.step(g, h, m, c.dt)
        return {"g": g.cpu().numpy(), "h": h.cpu().numpy(), "macros": told(m)}
    c = user_case(case, seed)
    if kind == "adjoint":
        # the whole run on the autograd tape: about 60 arrays of a face field a step
        if c.n_cells * 2 * c.n_dv * 8 * 60 * case["steps"] > 100e9 or not torch.cuda.is_available():
            return None
        return exact_adjoint(case, c)
    if not torch.cuda.is_available() and c.n_cells * c.n_dv * case["steps"] > 20_000_000:
        return None
    return exact_step(case, c)
