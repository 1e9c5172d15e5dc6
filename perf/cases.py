"""The timed cases: what programs on this framework spend their time in.

Three kinds of work:

* ``step``: ``Solver.step`` of one run in one of its forms (``fp64``,
  ``mixed64``, ``mixed``), from a flow that is already moving.  The FP64
  form's outputs are the state's own FP64 arrays on the device; the other two
  forms hand out the cell-centred float32 state (``pack_cells``), which is
  how plots, training data and judges take it.
* ``ensemble``: a window of steps of many small runs on one device, then the
  cell-centred state of every member, as training data is generated.
* ``unet``: the learned surrogate's network, the forward pass of a rollout or
  the forward and backward pass of a training batch (loss gradient to weight
  gradients).

Inputs come from the seed alone.  ``exact`` restates the same mathematics in
64 bits with plain torch.
"""

import ctypes
import math

import numpy as np
import torch

from pllcart3d_b200 import _lib
from pllcart3d_b200.ensemble import Ensemble
from pllcart3d_b200.params import Params, Workload
from pllcart3d_b200.solver import Solver
from pllcart3d_b200.surrogate import LAYERS, UNet, nnlib

F64 = torch.float64


def _step(name, form, nx, ny, nz, steps, nmvp=0):
    return {"name": name, "kind": "step", "form": form, "nx": nx, "ny": ny, "nz": nz, "steps": steps, "nmvp": nmvp}


def listed():
    return [
        # the smallest run, advanced one step at a time (a host loop that
        # looks at the state after every step): launches and latency
        _step("step-fp64-64x32x32", "fp64", 64, 32, 32, 1),
        # the window a rollout's judge runs between two looks at the state
        _step("window-fp64-128x64x64", "fp64", 128, 64, 64, 8),
        # the medium production run in plain FP64
        _step("step-fp64-256x128x128", "fp64", 256, 128, 128, 1),
        # a grid cut to an experiment's box, no extent a power of two
        _step("step-fp64-150x75x53", "fp64", 150, 75, 53, 2),
        # the non-monotonic viscosity law on a mid-sized odd box
        _step("step-fp64-nmvp-192x96x80", "fp64", 192, 96, 80, 1, 1),
        # the largest run, in the form that keeps c to 1e-5 over 1000 steps
        _step("step-mixed64-512x256x256", "mixed64", 512, 256, 256, 1),
        # the same run in the throughput form (FP32 state)
        _step("step-mixed-512x256x256", "mixed", 512, 256, 256, 1),
        # the throughput form on extents the tensor-core tiles do not divide
        _step("step-mixed-190x90x70", "mixed", 190, 90, 70, 2),
        # training data: members on the ensemble workload's four grids
        {"name": "ensemble-mixed-24", "kind": "ensemble", "members": 24, "steps": 4},
        # one window of a rollout
        {"name": "unet-forward-1x128x64x64", "kind": "unet", "batch": 1, "d": 128, "h": 64, "w": 64, "train": False},
        # one training batch
        {"name": "unet-train-8x128x64x64", "kind": "unet", "batch": 8, "d": 128, "h": 64, "w": 64, "train": True},
    ]


def draw(rng):
    pick = rng.random()
    if pick < 0.70:
        form = rng.choice(["fp64", "fp64", "mixed64", "mixed"])
        while True:
            nx = int(round(math.exp(rng.uniform(math.log(32), math.log(512)))))
            ny = int(round(math.exp(rng.uniform(math.log(24), math.log(256)))))
            nz = int(round(math.exp(rng.uniform(math.log(24), math.log(256)))))
            if rng.random() < 0.35:   # people like powers of two
                nx, ny, nz = (2 ** int(round(math.log2(n))) for n in (nx, ny, nz))
            if nx * ny * nz <= 8_000_000:
                break
        nmvp = 1 if form == "fp64" and rng.random() < 0.15 else 0
        return {"kind": "step", "form": form, "nx": nx, "ny": ny, "nz": nz, "steps": rng.randint(1, 4), "nmvp": nmvp}
    if pick < 0.82:
        return {"kind": "ensemble", "members": rng.randint(4, 24), "steps": rng.randint(1, 4)}
    d, h, w = rng.choice([(64, 32, 32), (64, 64, 64), (128, 64, 64), (96, 48, 64), (72, 40, 56)])
    return {"kind": "unet", "batch": rng.randint(1, 7), "d": d, "h": h, "w": w, "train": rng.random() < 0.5}


# ---- inputs -----------------------------------------------------------------

GRIDS = ((32, 32, 32), (64, 32, 32), (64, 64, 64), (128, 64, 64))


def _params(nx, ny, nz, nmvp, rng):
    """Physics in the measured workloads' ranges."""
    p = Params(Nx_cell_global=nx, Ny_cell_global=ny, Nz_cell_global=nz, Re=float(rng.uniform(100, 1000)),
               Pe=float(math.exp(rng.uniform(math.log(500), math.log(5000)))), Vratio=-float(rng.uniform(0.5, 3)),
               Fy=float(rng.uniform(0, 100)))
    return p.replace(Nmvp=1, Vratio=1.0) if nmvp else p


def _fields(p, rng):
    """(c, u, v, w) over the padded box, FP64 on the GPU where there is one:
    a fingered interface in a stream that already bends around it."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    NX, NY, NZ = p.nx + 6, p.ny + 2, p.nz + 2
    lx, ly, lz = p.X2 - p.X1, p.Y2 - p.Y1, p.Z2 - p.Z1
    x = (torch.arange(NX, dtype=F64, device=dev) - 3)[:, None, None] * p.dx     # faces, from the inlet
    y = (torch.arange(NY, dtype=F64, device=dev) - 1)[None, :, None] * p.dy     # faces, from the wall
    z = (torch.arange(NZ, dtype=F64, device=dev) - 1)[None, None, :] * p.dz
    xc, yc, zc = x + 0.5 * p.dx, y + 0.5 * p.dy, z + 0.5 * p.dz
    pi = math.pi
    eta = 0
    for _ in range(8):
        ky, kz = (int(k) for k in rng.integers(1, 5, 2))
        a, b = rng.uniform(0, 2 * pi, 2)
        eta = eta + 0.02 * torch.cos(2 * pi * ky * yc / ly + a) * torch.cos(2 * pi * kz * zc / lz + b)
    c = 0.5 * (1 - torch.tanh((xc - float(rng.uniform(0.9, 1.6)) - eta) / 0.05))
    u = torch.ones((NX, NY, NZ), dtype=F64, device=dev)
    v, w = torch.zeros_like(u), torch.zeros_like(u)
    for _ in range(3):
        kx, ky, kz = (int(k) for k in rng.integers(1, 4, 3))
        a = float(rng.uniform(0, 2 * pi))
        amp = rng.uniform(0.02, 0.08, 3)
        u += amp[0] * torch.sin(pi * kx * x / lx) * torch.cos(pi * ky * yc / ly + a) * torch.cos(pi * kz * zc / lz)
        v += amp[1] * torch.cos(pi * kx * xc / lx + a) * torch.sin(pi * ky * y / ly) * torch.cos(pi * kz * zc / lz)
        w += amp[2] * torch.cos(pi * kx * xc / lx + a) * torch.cos(pi * ky * yc / ly) * torch.sin(pi * kz * z / lz)
    # the inlet is a uniform stream; nothing crosses the walls
    u[:4] = 1.0
    v[:, 1], v[:, p.ny + 1] = 0.0, 0.0
    w[:, :, 1], w[:, :, p.nz + 1] = 0.0, 0.0
    return {"c": c, "u": u, "v": v, "w": w}


def _run_inputs(case, seed):
    rng = np.random.default_rng([int(seed), 1])
    p = _params(case["nx"], case["ny"], case["nz"], case["nmvp"], rng)
    return p, _fields(p, rng)


def _member_inputs(case, seed):
    out = []
    for m in range(case["members"]):
        rng = np.random.default_rng([int(seed), 2, m])
        p = _params(*GRIDS[m % len(GRIDS)], 0, rng)
        out.append((p, _fields(p, rng)))
    return out


def _net_inputs(case, seed):
    """Network weights (as bfloat16 holds them), input voxels, targets."""
    rng = np.random.default_rng([int(seed), 3])
    weights = {}
    for n, ci, co, k, act in LAYERS:
        w = rng.standard_normal((co, k ** 3, ci)) * math.sqrt(2.0 / (k ** 3 * ci)) * (1.0 if act else 0.1)
        w = torch.tensor(w, dtype=torch.float32).to(torch.bfloat16).to(torch.float32)
        weights[n] = (w.numpy(), (0.05 * rng.standard_normal(co)).astype(np.float32))
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    V = case["batch"] * case["d"] * case["h"] * case["w"]
    x = torch.zeros((V, 16), dtype=torch.float32, device="cuda")
    x[:, :4] = torch.randn((V, 4), generator=g, device="cuda")
    x[:, 4:6] = torch.rand((1, 2), generator=g, device="cuda")
    t = torch.zeros((V, 16), dtype=torch.float32, device="cuda")
    t[:, :4] = torch.randn((V, 4), generator=g, device="cuda")
    return weights, x.to(torch.bfloat16), t


STATE = ("c_old", "u_old", "v_old", "w_old", "u_pg", "v_pg", "w_pg", "phi")


class _DeviceArray:
    """A solver's array for torch, which keeps the solver as long as a tensor
    shows the array."""

    def __init__(self, owner, ptr, shape, strides):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "strides": strides, "typestr": "<f8", "data": (ptr, False),
                                         "version": 3}


def _state_views(s, seen):
    """The FP64 state's arrays on the device, as torch tensors (a field lives
    in one of two buffers by turns: `seen` keeps a view of each)."""
    L, out = _lib.lib(), []
    ptr, si, sj = ctypes.c_void_p(), ctypes.c_long(), ctypes.c_long()
    for f in STATE:
        code = L.pllgpu_device_field(s._h, _lib.FIELD_NAMES.index(f), ctypes.byref(ptr), ctypes.byref(si),
                                     ctypes.byref(sj))
        if code:
            raise _lib.PllGpuError(code, f)
        t = seen.get(ptr.value)
        if t is None:
            t = seen[ptr.value] = torch.as_tensor(
                _DeviceArray(s, ptr.value, s.shape, (8 * si.value, 8 * sj.value, 8)), device="cuda")
        out.append(t)
    return out


def prepare(case, seed):
    if case["kind"] == "step":
        p, f = _run_inputs(case, seed)
        s = Solver(p, precision=case["form"])
        s.load_ic({k: v.cpu().numpy() for k, v in f.items()})
        state = {"case": case, "solver": s}
        if case["form"] == "fp64":
            state["seen"] = {}
        else:
            state["cells"] = torch.empty((p.nx, p.ny, p.nz, 4), dtype=torch.float32, device="cuda")
        return state
    if case["kind"] == "ensemble":
        members = _member_inputs(case, seed)
        ens = Ensemble([Workload(f"member{m}", p) for m, (p, _) in enumerate(members)], precision="mixed")
        for s, (_, f) in zip(ens.members, members):
            for k, v in f.items():
                s.set(f"{k}_new", v.cpu().numpy())
        ens._check(_lib.lib().pllgpu_ensemble_start(ens._h), "ensemble_start")
        cells = [torch.empty((p.nx, p.ny, p.nz, 4), dtype=torch.float32, device="cuda") for p, _ in members]
        return {"case": case, "ensemble": ens, "cells": cells}
    weights, x, t = _net_inputs(case, seed)
    net = UNet(seed=0)
    net.load_state_dict(weights)
    return {"case": case, "net": net, "x": x, "target": t, "grad": torch.empty_like(t),
            "loss": torch.zeros(1, dtype=torch.float32, device="cuda"),
            "vol": (case["batch"], case["d"], case["h"], case["w"])}


def run(state):
    case = state["case"]
    if case["kind"] == "step":
        s = state["solver"]
        s.step(case["steps"])
        if case["form"] == "fp64":
            return _state_views(s, state["seen"])
        s.pack_cells(state["cells"].data_ptr())
        return state["cells"]
    if case["kind"] == "ensemble":
        state["ensemble"].step(case["steps"])
        for s, cells in zip(state["ensemble"].members, state["cells"]):
            s.pack_cells(cells.data_ptr())
        return state["cells"]
    net = state["net"]
    out = net.forward(state["x"], state["vol"])
    if not case["train"]:
        return out
    net.zero_grad()
    state["loss"].zero_()
    p = lambda a: ctypes.c_void_p(a.data_ptr())   # noqa: E731
    code = nnlib().pllnn_mse(p(out), p(state["target"]), out.numel(), 1.0 / (out.shape[0] * 4), p(state["grad"]),
                             p(state["loss"]), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if code:
        raise RuntimeError(f"mse failed ({code})")
    net.backward(state["grad"])
    return {"out": out, "grads": [g for c in net.layers.values() for g in (c.gw, c.gb)]}


# ---- what a pass cannot do without -------------------------------------------

def _step_work(cells, words):
    """Per step and cell: c, u, v, w, three pressure gradients and the old
    viscosity's source read once and written once, phi written, in each of
    the three substeps; the WENO5 passes (12 per substep, ~60 operations),
    the line solves (12, ~10) and the two transforms (~5 log2 n per axis)."""
    return {"bytes": 3.0 * 15 * words * cells, "flops": 3.0 * cells * (12 * 60 + 12 * 10 + 4 * 40)}


def work(case):
    if case["kind"] == "step":
        words = 4 if case["form"] == "mixed" else 8
        w = _step_work(case["nx"] * case["ny"] * case["nz"], words)
        return {k: v * case["steps"] for k, v in w.items()}
    if case["kind"] == "ensemble":
        cells = sum(math.prod(GRIDS[m % len(GRIDS)]) for m in range(case["members"]))
        return {k: v * case["steps"] for k, v in _step_work(cells, 4).items()}
    V = case["batch"] * case["d"] * case["h"] * case["w"]
    scale = {"e1": 1, "e2": 8, "e3": 64, "e4": 512, "d3": 64, "d2": 8, "d1": 1, "out": 1}
    fwd = sum(2.0 * V / scale[n] * ci * co * k ** 3 for n, ci, co, k, _ in LAYERS)
    acts = sum(2.0 * V / scale[n] * (ci + co) for n, ci, co, k, _ in LAYERS)
    if not case["train"]:
        return {"bytes": acts, "flops": fwd}
    first = 2.0 * V * 16 * 32 * 27   # the first layer passes no gradient on
    return {"bytes": 3 * acts, "flops": 3 * fwd - first}


# ---- the same mathematics in 64 bits ------------------------------------------

RK = ((8.0 / 15.0, 0.0), (5.0 / 12.0, -17.0 / 60.0), (3.0 / 4.0, -5.0 / 12.0))
C, U, V, W = range(4)
# ends of a line solve, (variable, axis): "n" mirrors the unknown (b += a),
# "r" reflects it about a wall face (b -= a), "0" is a fixed face
LOW = ("0nn", "0rn", "r0n", "rr0")
HIGH = ("0nn", "0rn", "00n", "0r0")


def _sh(a, axis, n):
    """a shifted so that element i holds a[i + n] (the ends wrap, unused)."""
    return torch.roll(a, -n, axis)


class _Exact:
    def __init__(self, p, f):
        self.p, self.h = p, (p.dx, p.dy, p.dz)
        self.n = (p.nx, p.ny, p.nz)
        first = ((3, 1, 1), (4, 1, 1), (3, 2, 1), (3, 1, 2))
        self.rng = [[(s, e) for s, e in zip(fs, (p.nx + 2, p.ny, p.nz))] for fs in first]
        self.q = [f[k].clone() for k in "cuvw"]
        self.H = [torch.zeros_like(f["c"]) for _ in range(4)]
        self.pg = [None] + [torch.zeros_like(f["c"]) for _ in range(3)]
        self.phi = torch.zeros_like(f["c"])
        self.ghosts(self.q)
        self.law = self.viscosity_law()
        self.mu = self.viscosity(self.q[C])
        self.cap = min(p.Timestep, 0.1 * p.Pe * min(self.h) ** 2)

    def box(self, v):
        return tuple(slice(s, e + 1) for s, e in self.rng[v])

    def viscosity_law(self):
        p = self.p
        if not p.Nmvp:
            return lambda c: torch.exp(p.Vratio * c)
        near = lambda a, h, n: min(range(1, n + 1), key=lambda i: (round(abs(a + (i - 0.5) * h), 12), i))   # noqa: E731
        line = self.q[C][3:p.nx + 3, near(p.Y1, p.dy, p.ny), near(p.Z1, p.dz, p.nz)].cpu().numpy()
        alpha = math.exp(p.Vratio)
        mum = p.Mum * alpha
        psi0, psi1 = math.asin(alpha / mum), math.pi - math.asin(1 / mum)
        em = (math.pi / 2 - psi0) / (psi1 - psi0)
        slope = lambda cm: ((1 - cm) - em) / ((1 - cm) * (em - 1))   # noqa: E731
        # the slopes at the two ends of the line (a first cell that is mixed
        # does not end the scan from its side); 0/0 in pure fluid ends the
        # bisection with its first halving
        i1 = next((i for i in range(1, p.nx) if abs(line[i]) > 1e-5), 0)
        i2 = next((i for i in range(p.nx - 1, 0, -1) if abs(line[i]) < 1 - 1e-5), 0)
        lo, hi, err = 0.1, 0.9, 1.0
        while err > 1e-5:
            cm = 0.5 * (lo + hi)
            eta = (1 + slope(cm)) * line / (1 + slope(cm) * line)
            mu = mum * np.sin(psi0 * (1 - eta) + psi1 * eta)
            with np.errstate(invalid="ignore", divide="ignore"):
                d = np.diff(mu) / np.diff(line)
            lam = (d[i1] + d[i2 - 1]) / (alpha + 1)
            lo, hi = (lo, cm) if lam > p.Lambda else (cm, hi)
            err = abs(lam - p.Lambda)
        a = slope(0.5 * (lo + hi))

        def law(c):
            eta = (1 + a) * c / (1 + a * c)
            return mum * torch.sin(psi1 * (1 - eta) + psi0 * eta)
        return law

    def viscosity(self, c):
        """At cell centres and at the xy, xz and yz edges."""
        m = lambda a, ax: a + _sh(a, ax, -1)   # noqa: E731
        return [self.law(c)] + [self.law(0.25 * m(m(c, a), b)) for a, b in ((0, 1), (0, 2), (1, 2))]

    def lower(self, mu, v, axis):
        """Coefficient of the lower neighbour; the upper one's is the same
        array one point on."""
        p, h = self.p, self.h[axis]
        if v == C:
            return torch.full_like(self.phi, 1.0 / (p.Pe * h * h))
        if axis == v - 1:
            return 2.0 / (p.Re * h * h) * _sh(mu[0], axis, -1)
        return 1.0 / (p.Re * h * h) * mu[axis + v - 1]   # the edge family of (axis, v - 1)

    def advect(self, v, axis, vel):
        """The velocity along `axis` at the points of variable v."""
        a = vel[axis + 1]
        if axis == v - 1:
            return a
        a = 0.5 * (a + _sh(a, axis, 1))
        return a if v == C else 0.5 * (a + _sh(a, v - 1, -1))

    def upwind(self, v, axis, q, vel, stale):
        """(advecting velocity) x (upwind derivative), moved to axis 0;
        `stale` are the second differences the previous axis left behind."""
        s, e = self.rng[v][axis]
        h = self.h[axis]
        box = list(self.box(v))
        box[axis] = slice(None)
        q = q[tuple(box)].movedim(axis, 0)
        vv = self.advect(v, axis, vel)[self.box(v)].movedim(axis, 0)
        d1 = torch.zeros_like(q)
        d1[:-1] = (q[1:] - q[:-1]) / h
        d2 = torch.zeros_like(q)
        for m in (s - 1, e + 1):
            if m < stale.numel():
                d2[m] = stale[m]
        d2[s:e + 1] = (d1[s:e + 1] - d1[s - 1:e]) / (2 * h)
        up = vv >= 0
        D = lambda t: d1[s + t:e + 1 + t]   # noqa: E731
        near = [torch.where(up, d2[s - 1:e], d2[s:e + 1]), torch.where(up, d2[s:e + 1], d2[s + 1:e + 2])]
        near = torch.where(near[0].abs() <= near[1].abs(), near[0], near[1])
        out = torch.where(up, D(-1) + near * h, D(0) - near * h)
        if e - s >= 4:
            D = lambda t: d1[s + 2 + t:e - 1 + t]   # noqa: E731
            a = up[2:-2]
            out[2:-2] = self.weno([torch.where(a, D(t - 3), D(2 - t)) for t in range(5)])
        last = torch.zeros_like(stale) if stale.numel() >= q.shape[0] else stale.new_zeros(q.shape[0])
        last[:stale.numel()] = stale
        last[s:e + 1] = d2[s:e + 1].reshape(e - s + 1, -1)[:, -1]
        return (vv * out).movedim(0, axis), last

    @staticmethod
    def weno(v):
        c = [(2 * v[0] - 7 * v[1] + 11 * v[2]) / 6, (-v[1] + 5 * v[2] + 2 * v[3]) / 6, (2 * v[2] + 5 * v[3] - v[4]) / 6]
        s = [13 / 12 * (v[0] - 2 * v[1] + v[2]) ** 2 + 0.25 * (v[0] - 4 * v[1] + 3 * v[2]) ** 2,
             13 / 12 * (v[1] - 2 * v[2] + v[3]) ** 2 + 0.25 * (v[1] - v[3]) ** 2,
             13 / 12 * (v[2] - 2 * v[3] + v[4]) ** 2 + 0.25 * (3 * v[2] - 4 * v[3] + v[4]) ** 2]
        eps = v[0] * v[0]
        for x in v[1:]:
            eps = torch.maximum(eps, x * x)
        eps = 1e-6 * eps + 1e-99
        a = [g / (x + eps) ** 2 for g, x in zip((0.1, 0.6, 0.3), s)]
        at = a[0] + a[1] + a[2]
        return sum(x / at * y for x, y in zip(a, c))

    def explicit(self, v, vel, mu):
        box, q = self.box(v), self.q[v]
        stale = q.new_zeros(0)
        total = 0
        for axis in range(3):
            part, stale = self.upwind(v, axis, q, vel, stale)
            total = total - part
        if v != C:   # cross stress: d/dx_a (mu du_a/dx_v)
            for axis in range(3):
                if axis == v - 1:
                    continue
                s = mu[axis + v - 1] * (vel[axis + 1] - _sh(vel[axis + 1], v - 1, -1))
                total = total + ((_sh(s, axis, 1) - s) / (self.p.Re * self.h[axis] * self.h[v - 1]))[box]
        H = torch.zeros_like(q)
        H[box] = total
        return H

    @staticmethod
    def thomas(a, b, c, r):
        """Lines along axis 0, overwritten."""
        cc, ib = torch.empty_like(c), 1.0 / b[0]
        cc[0], r[0] = c[0] * ib, r[0] * ib
        for i in range(1, r.shape[0]):
            ib = 1.0 / torch.addcmul(b[i], cc[i - 1], a[i], value=-1)
            torch.mul(c[i], ib, out=cc[i])
            torch.mul(torch.addcmul(r[i], r[i - 1], a[i], value=-1), ib, out=r[i])
        for i in range(r.shape[0] - 2, -1, -1):
            r[i].addcmul_(cc[i], r[i + 1], value=-1)
        return r

    def advance(self, v, vel, cn, mu_old, mu_new, dt, g, r, vb):
        """One variable's substep; returns its new field and explicit term."""
        p, box, q = self.p, self.box(v), self.q[v]
        alpha = g + r
        H = self.explicit(v, vel, mu_old)
        diff = 0
        for axis in range(3):
            a = self.lower(mu_old, v, axis)
            flux = a * (_sh(q, axis, -1) - q)
            diff = diff + (flux - _sh(flux, axis, 1))[box]
        S = g * H[box] + r * self.H[v][box] + alpha * diff
        if v != C:
            force = -self.pg[v] / p.Re
            if v != W:
                force = force - (p.Fx, p.Fy)[v - 1] / p.Re * 0.5 * (cn + _sh(cn, v - 1, -1))
            S = S + alpha * force[box]
        S = dt * S
        fac = 0.5 * dt * alpha
        out = self.n[0] + 3   # the outflow face or the ghost cell behind it
        H[out][box[1:]] = (-vb * (q[out] - q[out - 1]) / p.dx)[box[1:]]
        boun = dt * (g * H[out] + r * self.H[v][out])
        for axis in (1, 2, 0):
            a = self.lower(mu_new, v, axis)
            up = -fac * _sh(a, axis, 1)[box].movedim(axis, 0)
            a = -fac * a[box].movedim(axis, 0)
            b = 1.0 - a - up
            for row, side, lo in ((0, a, LOW), (-1, up, HIGH)):
                if lo[v][axis] == "n":
                    b[row] += side[row]
                elif lo[v][axis] == "r":
                    b[row] -= side[row]
            x = S.movedim(axis, 0).contiguous()
            if axis == 0:
                x[-1] -= up[-1] * boun[box[1:]]
            S = self.thomas(a, b, up, x).movedim(0, axis)
        new = q.clone()
        new[box] = q[box] + S
        new[out][box[1:]] = (q[out] + boun)[box[1:]]
        if v == C:
            i, j = slice(3, self.n[0] + 3), self.n[1]
            k = self.n[2]
            new[i, 0, 1:-1], new[i, j + 1, 1:-1] = new[i, 1, 1:-1], new[i, j, 1:-1]
            new[i, :, 0], new[i, :, k + 1] = new[i, :, 1], new[i, :, k]
        return new, H

    def ghosts(self, q):
        _, u, v, w = q
        nx, ny, nz = self.n
        i, j, k = slice(3, nx + 3), slice(1, ny + 1), slice(1, nz + 1)
        for a in (u, v):
            a[i, j, 0], a[i, j, nz + 1] = a[i, j, 1], a[i, j, nz]
        for a in (u, w):
            a[i, 0, k], a[i, ny + 1, k] = -a[i, 1, k], -a[i, ny, k]
        for a in (v, w):
            a[2, j, k] = -a[3, j, k]

    def dct(self, n, inverse):
        """Matrix of the cosine transform (its inverse) of n points."""
        i = torch.arange(n, dtype=F64, device=self.phi.device)
        m = torch.cos(math.pi * i[:, None] * (i[None, :] + 0.5) / n)   # [mode][point]
        if not inverse:
            return 2.0 * m
        m = m.T / n
        return torch.cat([m[:, :1] * 0.5, m[:, 1:]], 1)

    def poisson(self, src):
        p = self.p
        nx, ny, nz = self.n
        hat = torch.einsum("ab,xbc,dc->xad", self.dct(ny, 0), src, self.dct(nz, 0))
        k = [2.0 * (torch.cos(math.pi * torch.arange(n, dtype=F64, device=src.device) / n) - 1.0) / h ** 2
             for n, h in ((ny, p.dy), (nz, p.dz))]
        d = 1.0 / p.dx ** 2
        b = (-2.0 * d + k[0][:, None] + k[1][None, :]).expand(nx, ny, nz).clone()
        b[0] += d
        last = b[-1, 0, 0].clone()
        b[-1] += d
        b[-1, 0, 0] = last   # the constant mode is fixed to 0 behind the outflow
        off = torch.full_like(b, d)
        hat = self.thomas(off, b, off, hat.contiguous())
        return torch.einsum("ab,xbc,dc->xad", self.dct(ny, 1), hat, self.dct(nz, 1))

    def flux(self, u, i):
        """Trapezoid over the cell centres of a face plane."""
        a = u[i, 1:-1, 1:-1]
        a = 0.5 * self.h[2] * (a[:, 1:] + a[:, :-1]).sum(1)
        return 0.5 * self.h[1] * (a[1:] + a[:-1]).sum()

    def substep(self, dt, g, r):
        p = self.p
        nx, ny, nz = self.n
        alpha = g + r
        face = self.q[U][nx + 2, 1:-1, 1:-1].reshape(-1)
        vb = face[face.abs().argmax()]
        new, H = [None] * 4, [None] * 4
        new[C], H[C] = self.advance(C, self.q, None, self.mu, self.mu, dt, g, r, vb)
        mu = self.viscosity(new[C])
        for v in (U, V, W):
            new[v], H[v] = self.advance(v, self.q, new[C], self.mu, mu, dt, g, r, vb)
        cell = self.box(C)
        div = sum((_sh(new[a + 1], a, 1) - new[a + 1])[cell] / self.h[a] for a in range(3))
        phi = self.phi
        phi[cell] = self.poisson(p.Re / (dt * alpha) * div)
        i, j, k = cell
        phi[i, j, 0], phi[i, j, nz + 1] = phi[i, j, 1], phi[i, j, nz]
        phi[i, 0, k], phi[i, ny + 1, k] = phi[i, 1, k], phi[i, ny, k]
        phi[2, j, k], phi[nx + 3, j, k] = phi[3, j, k], phi[nx + 2, j, k]
        grad = [None] + [(phi - _sh(phi, a, -1)) / self.h[a] for a in range(3)]
        for v in (U, V, W):
            box = self.box(v)
            new[v][box] -= dt * alpha / p.Re * grad[v][box]
        lack = (self.flux(new[U], 3) - self.flux(new[U], nx + 3)) / ((p.Y2 - p.Y1) * (p.Z2 - p.Z1))
        new[U][nx + 3, 1:-1, 1:-1] += lack
        self.ghosts(new)
        for v in (U, V, W):
            box, lap = self.box(v), 0
            for axis in range(3):
                f = self.lower(mu, v, axis) * (_sh(grad[v], axis, -1) - grad[v])
                lap = lap + f - _sh(f, axis, 1)
            self.pg[v][box] += (grad[v] - 0.5 * dt * alpha * lap)[box]
        self.q, self.H, self.mu = new, H, mu

    def step(self):
        mid = [0.5 * (self.q[a + 1] + _sh(self.q[a + 1], a, 1)).abs()[self.box(C)] / self.h[a]
               for a in range(3)]
        dt = min(self.cap, self.p.CFLmax / float((mid[0] + mid[1] + mid[2]).max()))
        for g, r in RK:
            self.substep(dt, g, r)

    def cells(self):
        """(u, v, w, c) at the cell centres."""
        return torch.stack([0.5 * (self.q[a + 1] + _sh(self.q[a + 1], a, 1))[self.box(C)] for a in range(3)]
                           + [self.q[C][self.box(C)]], -1)


def _exact_net(case, seed):
    weights, x, t = _net_inputs(case, seed)
    B, D, H, Wd = case["batch"], case["d"], case["h"], case["w"]
    par = {n: [torch.tensor(a, dtype=F64, device="cuda").requires_grad_(case["train"]) for a in wb]
           for n, wb in weights.items()}

    def conv(n, y, act=True):
        w, b = par[n]
        k = round(w.shape[1] ** (1 / 3))
        w = w.reshape(w.shape[0], k, k, k, -1).permute(0, 4, 1, 2, 3)
        z = torch.nn.functional.conv3d(y, w, b, padding=k // 2)
        return torch.nn.functional.leaky_relu(z, 0.1) if act else z

    pool = lambda y: torch.nn.functional.avg_pool3d(y, 2)   # noqa: E731
    join = lambda y, skip: torch.cat([y.repeat_interleave(2, 2).repeat_interleave(2, 3).repeat_interleave(2, 4),   # noqa: E731
                                      skip], 1)
    e1 = conv("e1", x.to(F64).reshape(B, D, H, Wd, 16).permute(0, 4, 1, 2, 3))
    e2 = conv("e2", pool(e1))
    e3 = conv("e3", pool(e2))
    d3 = conv("d3", join(conv("e4", pool(e3)), e3))
    d1 = conv("d1", join(conv("d2", join(d3, e2)), e1))
    out = conv("out", d1, False).permute(0, 2, 3, 4, 1).reshape(-1, 16)
    if not case["train"]:
        return out
    # the loss is the mean over the four channels that are used
    loss = (out - t.to(F64)).square().sum() / (out.shape[0] * 4)
    loss.backward()
    return {"out": out.detach(), "grads": [a.grad for n, *_ in LAYERS for a in par[n]]}


def exact(case, seed):
    if case["kind"] == "step":
        e = _Exact(*_run_inputs(case, seed))
        for _ in range(case["steps"]):
            e.step()
        return [*e.q, *e.pg[1:], e.phi] if case["form"] == "fp64" else e.cells()
    if case["kind"] == "ensemble":
        out = []
        for p, f in _member_inputs(case, seed):
            e = _Exact(p, f)
            for _ in range(case["steps"]):
                e.step()
            out.append(e.cells())
        return out
    return _exact_net(case, seed)
