"""The work that programs built on this solver have it do, as timed cases.

Each case is one call pattern of the public interface (tnsgpu.solver, tnsgpu.batch and the
adjoint entry points of the C ABI) on a mesh family and size the solver's configurations,
tests and benchmark use:

  solve      a device-resident FP64 loop: a state in device memory is loaded into the
             handle, advanced by some RK4 iterations, and copied back to device memory.
  coupled    a host program's step: page-locked state in, some iterations, the new state (in
             FP64 with the residual record) out, one wait at the end.  FP64 or mixed precision.
  general    a mesh in a grid generator's own numbering (not one i x j block): upload, some
             iterations (in FP64 with a residual record), download.  FP64 or mixed precision.
  batch      a parameter sweep: several ramp cases advanced together.
  adjoint    the reverse sweep of a gradient: a recorded primal and its reverse steps with
             the sensitivities ("transient"), or repeated steps at one state ("fixed").
  time_step  the allocation-free time step on a state in device memory.

``exact`` restates the scheme in FP64 torch arithmetic (one structured block, BC types
2-6), independent of the library.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "2d-turbulent-navier-stokes_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from tnsgpu import _lib, cases as meshes, formats  # noqa: E402
from tnsgpu.batch import Batch  # noqa: E402
from tnsgpu.solver import Solver, make_params  # noqa: E402

F64 = torch.float64


# ------------------------------------------------------------------------------- cases

def listed():
    return [
        # the example case of the reference's repository: a small solve, bound by latency
        {"name": "nozzle2d_115x50", "kind": "solve", "family": "nozzle2d", "ni": 115, "nj": 50, "local": 1, "iters": 10},
        # the smallest sweep case as one step of a coupled host program: one iteration a call
        {"name": "coupled_ramp_96x32", "kind": "coupled", "family": "ramp", "ni": 96, "nj": 32, "local": 1,
         "precision": 0, "iters": 1},
        # a time-accurate run (one global time step) on an odd-sized mesh
        {"name": "ramp_201x67_global_dt", "kind": "solve", "family": "ramp", "ni": 201, "nj": 67, "local": 0, "iters": 10},
        # the mid-size ramp, FP64
        {"name": "ramp_512x192", "kind": "solve", "family": "ramp", "ni": 512, "nj": 192, "local": 1, "iters": 10},
        # the benchmark's workload: axisymmetric nozzle + plume, FP64
        {"name": "nozzle_plume_1024x384", "kind": "solve", "family": "plume", "ni": 1024, "nj": 384, "local": 1,
         "iters": 10},
        # the same in mixed precision, driven from host memory
        {"name": "mixed_plume_1024x384", "kind": "coupled", "family": "plume", "ni": 1024, "nj": 384, "local": 1,
         "precision": 1, "iters": 10},
        # a large injecting port channel (type-6 walls: a port sum before every stage)
        {"name": "port_2048x768", "kind": "solve", "family": "port", "ni": 2048, "nj": 768, "local": 1, "iters": 4},
        # meshes in a generator's numbering: the general path in both precisions
        {"name": "general_plume_512x192", "kind": "general", "family": "plume", "ni": 512, "nj": 192, "local": 1,
         "precision": 0, "iters": 30},
        {"name": "general_mixed_ramp_256x96", "kind": "general", "family": "ramp", "ni": 256, "nj": 96, "local": 1,
         "precision": 1, "iters": 20},
        # a parameter sweep of ramp cases in mixed precision under the schedule tuning picks
        {"name": "sweep_16_mixed", "kind": "batch", "members": 16, "precision": 1, "schedule": 2, "iters": 20},
        # the gradient workload: record the primal, reverse it with all sensitivities
        {"name": "adjoint_ramp_512x192", "kind": "adjoint", "mode": "transient", "family": "ramp", "ni": 512, "nj": 192,
         "local": 1, "iters": 6},
        # the allocation-free time step of a host with its own state arrays
        {"name": "time_step_1572864", "kind": "time_step", "cells": 1572864},
    ]


# most cell-iterations a drawn case may ask for, by kind (the listed ones' cost)
_MOST = {"solve": 4.0e6, "coupled": 6.0e6, "general": 2.5e6, "adjoint": 5.0e5}


def _size(rng, lo, hi):
    """A mesh with lo .. hi cells (uniform in the logarithm), 1 to 4 times as long as high."""
    cells, aspect = math.exp(rng.uniform(math.log(lo), math.log(hi))), rng.uniform(1.0, 4.0)
    nj = max(6, int(round(math.sqrt(cells / aspect))))
    return max(8, int(round(cells / nj))), nj


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "coupled", "coupled", "general", "general", "batch", "adjoint",
                       "time_step"])
    if kind == "time_step":
        return {"kind": kind, "cells": int(math.exp(rng.uniform(math.log(5.0e3), math.log(6.0e6))))}
    if kind == "batch":
        return {"kind": kind, "members": rng.randint(4, 16), "precision": rng.randint(0, 1),
                "schedule": rng.choice([0, 1, 2]), "iters": rng.randint(5, 12)}
    family = rng.choice(["ramp", "plume", "nozzle2d", "port"])
    if kind == "adjoint":
        ni, nj = _size(rng, 2.0e3, 1.0e5)
        iters = max(1, min(8, int(_MOST[kind] / (ni * nj))))
        return {"kind": kind, "mode": rng.choice(["transient", "fixed"]), "family": family, "ni": ni, "nj": nj,
                "local": 1, "iters": rng.randint(1, iters)}
    ni, nj = _size(rng, 1.0e3, {"solve": 1.0e6, "coupled": 5.0e5, "general": 1.5e5}[kind])
    iters = max(1, min(20, int(_MOST[kind] / (ni * nj))))
    case = {"kind": kind, "family": family, "ni": ni, "nj": nj, "local": rng.choice([1, 1, 1, 0]),
            "iters": rng.randint(1, iters)}
    if kind != "solve":
        case["precision"] = rng.randint(0, 1)
        if case["precision"]:
            case["iters"] = min(case["iters"], 2 if family == "port" else 10)
    return case


# ------------------------------------------------------------------------------ inputs

def _setup(family, ni, nj, local):
    if family == "ramp":
        mesh, flow = meshes.ramp_mesh(ni, nj), meshes.ramp_flow()
    elif family == "plume":
        mesh, flow = meshes.nozzle_plume_mesh(ni, nj), meshes.nozzle_plume_flow()
    elif family == "nozzle2d":
        mesh, flow = meshes.nozzle_2d_mesh(ni, nj), meshes.nozzle_2d_flow()
    else:
        mesh, flow = meshes.port_mesh(ni, nj), meshes.port_flow()
    flow.local = local
    return mesh, flow


def _state(flow, ni, nj, seed):
    """A developing flow, [5, ni*nj] on the GPU: the cold start's pressure and temperature
    with pressure waves of 1e-3 and a little noise, a sheared velocity with waves, and an
    eddy viscosity that rises from the free-stream value near the boundaries to some 30
    times it inside."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 17)
    rand = lambda *s: torch.rand(*s, generator=g, device="cuda", dtype=F64)
    base = formats.cold_state(flow, 1)[:, 0]
    rho0, u0, r0 = base[0], base[1] / base[0], base[4] / base[0]
    e0 = base[3] / base[0] - 0.5 * u0 * u0
    x = ((torch.arange(ni, device="cuda", dtype=F64) + 0.5) / ni)[:, None]
    y = ((torch.arange(nj, device="cuda", dtype=F64) + 0.5) / nj)[None, :]
    ph = rand(8)
    wave = lambda k, a, b: torch.sin(2.0 * math.pi * (k * x + ph[a])) * torch.sin(math.pi * (k * y + ph[b]))
    u = u0 * (0.6 + 1.6 * y * (1.0 - y) + 0.2 * wave(2.0, 0, 1))
    v = 0.1 * u0 * wave(3.0, 2, 3)
    rho = rho0 * (1.0 + 1.0e-3 * wave(2.0, 6, 7) + 1.0e-5 * (2.0 * rand(ni, nj) - 1.0))
    r = r0 * (1.0 + 60.0 * y * (1.0 - y) * (1.0 + wave(1.0, 4, 5)) * (1.0 + 0.05 * rand(ni, nj)))
    c = torch.stack([rho, rho * u, rho * v, rho * (e0 + 0.5 * (u * u + v * v)), rho * r])
    return c.reshape(5, -1).contiguous()


_streams = []


def _stream():
    """The program's one working stream."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0]


def _pinned(*shape):
    return torch.empty(shape, dtype=F64, pin_memory=True)


def _ptrs(t):
    return [t[k].data_ptr() for k in range(5)]


def _sweep(case):
    """The first cases of the benchmark's sweep (96x32 .. 512x192)."""
    return meshes.ramp_sweep(64, seed=0)[:case["members"]]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "time_step":
        n = case["cells"]
        flow = meshes.ramp_flow()
        nj = max(d for d in range(1, 200) if n % d == 0)
        q = _state(flow, n // nj, nj, seed)
        g = torch.Generator(device="cuda").manual_seed(int(seed) + 5)
        cfldl = flow.cfl * 10.0 ** (-5.0 + 2.0 * torch.rand(n, generator=g, device="cuda", dtype=F64))
        return {"case": case, "lib": _lib.load(), "params": make_params(flow, formats.rinit_cold(flow)), "q": q,
                "cfldl": cfldl, "dt": torch.empty(n, device="cuda", dtype=F64),
                "dtmin": torch.empty(1, device="cuda", dtype=F64)}
    if kind == "batch":
        solvers, ins, outs = [], [], []
        for k, c in enumerate(_sweep(case)):
            mesh, flow = c.mesh(), c.flow()
            s = Solver(mesh, flow, formats.rinit_cold(flow), precision=case["precision"])
            ins.append(_pinned(5, mesh.neles))
            outs.append(_pinned(5, mesh.neles))
            ins[-1].copy_(_state(flow, c.nx, c.ny, seed * 100 + k))
            s.upload(ins[-1].numpy())
            solvers.append(s)
        b = Batch(solvers, schedule=case["schedule"])
        b.prepare()
        return {"case": case, "batch": b, "solvers": solvers, "ins": ins, "outs": outs}
    ni, nj = case["ni"], case["nj"]
    mesh, flow = _setup(case["family"], ni, nj, case["local"])
    rinit = formats.rinit_cold(flow)
    q = _state(flow, ni, nj, seed)
    st = {"case": case}
    if kind == "general":
        mesh, perm = meshes.renumbered_mesh(mesh, seed=3)
        host = np.empty((5, ni * nj))
        host[:, perm] = q.cpu().numpy()
        st["solver"] = s = Solver(mesh, flow, rinit, precision=case["precision"])
        st["q"] = host
        s.upload(host)
        s.prepare()
        return st
    st["solver"] = s = Solver(mesh, flow, rinit, precision=case.get("precision", 0))
    st["stream"] = stream = _stream()
    s.set_stream(stream.cuda_stream)
    if kind == "coupled":
        st["in"], st["out"], st["record"] = _pinned(5, ni * nj), _pinned(5, ni * nj), _pinned(5)
        st["in"].copy_(q)
        s.upload(st["in"].numpy())
        s.prepare()
        return st
    st["q"] = q
    if kind == "solve":
        st["out"] = torch.empty_like(q)
        s.upload(q.cpu().numpy())
        s.prepare()
        return st
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 11)
    scale = 1.0 / q.abs().amax(dim=1, keepdim=True)  # an objective's derivative: each component at its own scale
    st["seed_lam"] = torch.randn(5, ni * nj, generator=g, device="cuda", dtype=F64) * scale
    st["lam"] = torch.empty_like(q)
    n = case["iters"]
    if case["mode"] == "transient":
        st["states"] = torch.empty((n + 1, 5, ni * nj), device="cuda", dtype=F64)
        st["states"][0].copy_(q)
        st["records"] = torch.empty((n, s.adjoint_record_size()), device="cuda", dtype=F64)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    n = case.get("iters", 0)
    if kind == "time_step":
        p = lambda t: ctypes.c_void_p(t.data_ptr())
        rc = st["lib"].tns_time_step_noalloc(p(st["q"]), p(st["cfldl"]), case["cells"], ctypes.byref(st["params"]),
                                             p(st["dt"]), p(st["dtmin"]),
                                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc:
            raise _lib.TnsError(rc, "tns_time_step_noalloc")
        return st["dt"], st["dtmin"]
    if kind == "batch":
        for s, q in zip(st["solvers"], st["ins"]):
            s.upload_async(_ptrs(q))
        for s in st["solvers"]:
            s.synchronize()
        rec = st["batch"].run(n, 0 if case["precision"] else n).records
        for s, q in zip(st["solvers"], st["outs"]):
            s.download_async(_ptrs(q))
        for s in st["solvers"]:
            s.synchronize()
        return st["outs"] if case["precision"] else (st["outs"], np.concatenate(rec))
    s = st["solver"]
    if kind == "solve":
        s.state_from_device(st["q"].data_ptr())
        s.enqueue(n)
        s.state_to_device(st["out"].data_ptr())
        return st["out"]
    if kind == "coupled":
        s.upload_async(_ptrs(st["in"]))
        if case["precision"]:
            s.enqueue(n)
        else:
            if n > 1:
                s.enqueue(n - 1)
            s.enqueue_monitored(st["record"].data_ptr())
        s.download_async(_ptrs(st["out"]))
        s.synchronize()
        return st["out"] if case["precision"] else (st["out"], st["record"])
    if kind == "general":
        s.upload(st["q"])
        rec = s.run(n, 0 if case["precision"] else n)
        return s.download() if case["precision"] else (s.download(), rec)
    lam = st["lam"]
    if case["mode"] == "transient":
        q, rec = st["states"], st["records"]
        with torch.cuda.stream(st["stream"]):
            lam.copy_(st["seed_lam"])
        for k in range(n):
            s.adjoint_record(q[k].data_ptr(), q[k + 1].data_ptr(), rec[k].data_ptr())
        for k in range(n - 1, -1, -1):
            s.adjoint_step(q[k].data_ptr(), lam.data_ptr(), True, rec_ptr=rec[k].data_ptr())
        return lam, q[n], s.adjoint_sensitivities()
    with torch.cuda.stream(st["stream"]):
        lam.copy_(st["seed_lam"])
    for k in range(n):  # lambda <- dJ/dQ + lambda dG/dQ at one state
        s.adjoint_step(st["q"].data_ptr(), lam.data_ptr(), False, frozen=k > 0)
        with torch.cuda.stream(st["stream"]):
            lam.add_(st["seed_lam"])
    return lam


def work(case):
    """Bytes and operations a pass cannot do without.  An iteration reads the state, the node
    coordinates and CFL*DL of every cell and writes the new state: 104 bytes a cell; its
    arithmetic is some 2700 operations a cell (four stages of about 450, the viscous faces
    and the dissipation).  A reverse step also reads its record of 25 doubles a cell and
    updates the adjoint state and, where asked, 17 doubles of sensitivities."""
    kind = case["kind"]
    if kind == "time_step":
        return {"bytes": 48.0 * case["cells"] + 8.0 * case["cells"], "flops": 20.0 * case["cells"]}
    if kind == "batch":
        cells = float(sum(c.nx * c.ny for c in _sweep(case)))
    else:
        cells = float(case["ni"] * case["nj"])
    n = case["iters"]
    if kind == "adjoint":
        if case["mode"] == "transient":
            return {"bytes": n * cells * (104.0 + 200.0 + 200.0 + 80.0 + 272.0), "flops": n * cells * 12000.0}
        return {"bytes": n * cells * (200.0 + 120.0), "flops": n * cells * 6000.0}
    return {"bytes": n * cells * 104.0, "flops": n * cells * 2700.0}


# ------------------------------------------------------------------- the scheme in FP64

CMU, ALPHA_T, BETA_T, SUTH = 0.09, 0.00052, 0.2, 0.00000011848
ALPHA_RK = (0.25, 1.0 / 3.0, 0.5, 1.0)


def _sqrt(x):
    """sqrt with a zero derivative at zero."""
    pos = x > 0
    return torch.where(pos, torch.sqrt(torch.where(pos, x, torch.ones_like(x))), torch.zeros_like(x))


def _dmax(a, b):
    return torch.where(a >= b, a, b)


def _around(a):
    """The neighbours across faces 1..4 (j-, i+, j+, i-) of a padded field's inner cells."""
    return a[..., 1:-1, :-2], a[..., 2:, 1:-1], a[..., 1:-1, 2:], a[..., :-2, 1:-1]


def _replicate(a):
    a = torch.cat([a[..., :1, :], a, a[..., -1:, :]], dim=-2)
    return torch.cat([a[..., :, :1], a, a[..., :, -1:]], dim=-1)


class _Scheme:
    """One RK4 iteration on one i x j block, cells [ni, nj], in FP64."""

    def __init__(self, mesh, flow, rinit):
        ni, nj = mesh.shape
        self.ni, self.nj, self.flow = ni, nj, flow
        dev = dict(device="cuda", dtype=F64)
        x = torch.tensor(mesh.x.reshape(ni + 1, nj + 1), **dev)
        y = torch.tensor(mesh.y.reshape(ni + 1, nj + 1), **dev)
        self.rr = 8314.0 / flow.amol
        self.cv = self.rr / (flow.gama - 1.0)
        self.cp = self.cv * flow.gama
        self.s0 = flow.p0 / (flow.p0 / (self.rr * flow.t0)) ** flow.gama
        self.rtol = rinit * flow.rtred
        self.amu_c = SUTH * math.sqrt(flow.amol)
        axi = flow.iaxis == 1
        X = [x[:-1, :-1], x[1:, :-1], x[1:, 1:], x[:-1, 1:]]
        Y = [y[:-1, :-1], y[1:, :-1], y[1:, 1:], y[:-1, 1:]]
        xc, yc = (X[0] + X[1] + X[2] + X[3]) * 0.25, (Y[0] + Y[1] + Y[2] + Y[3]) * 0.25
        self.sx, self.sy, self.faces, dl = [], [], [], None
        for k in range(4):
            xa, ya, xb, yb = X[k], Y[k], X[(k + 1) % 4], Y[(k + 1) % 4]
            h = (ya + yb) * 0.5 if axi else 1.0
            self.sx.append((yb - ya) * h)
            self.sy.append(-(xb - xa) * h)
            self.faces.append((xa, ya, xb, yb))
            d = torch.sqrt((xa - xb) ** 2 + (ya - yb) ** 2)
            dl = d if dl is None else torch.minimum(dl, d)
        self.dl = dl
        vol = 0.5 * ((X[2] - X[0]) * (Y[3] - Y[1]) - (X[3] - X[1]) * (Y[2] - Y[0]))
        self.vol = (vol * yc if axi else vol).abs()
        # centroids, the ghosts' mirrored in their faces
        self.xc, self.yc = _replicate(xc), _replicate(yc)
        mid = lambda a, k: 0.5 * (a[k] + a[(k + 1) % 4])
        inner, ring = slice(1, -1), [(slice(1, -1), 0), (-1, slice(1, -1)), (slice(1, -1), -1), (0, slice(1, -1))]
        at = [(slice(None), 0), (-1, slice(None)), (slice(None), -1), (0, slice(None))]
        for k in range(4):
            self.xc[ring[k]] = 2.0 * mid(X, k)[at[k]] - xc[at[k]]
            self.yc[ring[k]] = 2.0 * mid(Y, k)[at[k]] - yc[at[k]]
        self.inner = (inner, inner)
        # ghosts, sides 1..4 one after another: parent, the cell opposite, padded place, type
        i, j = np.arange(ni), np.arange(nj)
        full = lambda n, v: np.full(n, v)
        par = [(i, full(ni, 0)), (full(nj, ni - 1), j), (i, full(ni, nj - 1)), (full(nj, 0), j)]
        opp = [(i, full(ni, 1)), (full(nj, ni - 2), j), (i, full(ni, nj - 2)), (full(nj, 1), j)]
        pad = [(i + 1, full(ni, 0)), (full(nj, ni + 1), j + 1), (i + 1, full(ni, nj + 1)), (full(nj, 0), j + 1)]
        flat = lambda ps, w: torch.tensor(np.concatenate([a * w + b for a, b in ps]), device="cuda")
        self.g_par, self.g_opp, self.g_pad = flat(par, nj), flat(opp, nj), flat(pad, nj + 2)
        first = np.cumsum([0, ni, nj, ni])  # first ghost of each side
        p0 = mesh.nparent - 1
        where = first[mesh.nside - 1] + np.where(mesh.nside % 2 == 1, p0 // nj, p0 % nj)
        gtype, line, inj = (np.zeros(2 * (ni + nj), t) for t in (np.int64, np.int64, np.float64))
        gtype[where], line[where] = mesh.ntype, np.arange(mesh.nghosts)
        inj[where] = 1.0 if mesh.inj_scale is None else mesh.inj_scale
        self.g_type, self.g_inj = torch.tensor(gtype, device="cuda"), torch.tensor(inj, **dev)
        self.types = set(int(t) for t in gtype)
        # nodal averages: every boundary node has two ghosts, visited in bc.in order
        pair = {}
        for s in range(4):
            for k in range((ni, nj, ni, nj)[s]):
                a, b = par[s][0][k], par[s][1][k]
                n = [(a, b), (a + 1, b), (a + 1, b + 1), (a, b + 1)]
                for q in (n[s], n[(s + 1) % 4]):
                    pair.setdefault(q, []).append(first[s] + k)
        node, g1, g2 = [], [], []
        for (a, b), g in pair.items():
            g.sort(key=lambda v: line[v])
            node.append(a * (nj + 1) + b)
            g1.append(g[0])
            g2.append(g[1])
        it = lambda v: torch.tensor(np.asarray(v, np.int64), device="cuda")
        self.b_node, self.b_g = it(node), (it(g1), it(g2))
        cells = torch.zeros((ni + 2, nj + 2), **dev)
        cells[self.inner] = 1.0
        self.is_cell = cells
        count = self._four(cells).reshape(-1)
        count[self.b_node] += 2.0
        self.count = count.reshape(ni + 1, nj + 1)

    @staticmethod
    def _four(a):
        return a[..., :-1, :-1] + a[..., :-1, 1:] + a[..., 1:, :-1] + a[..., 1:, 1:]

    def amu(self, t):
        return self.amu_c * t ** 0.6

    @staticmethod
    def _set(u, v, t, p, rho, c4, ri, f5, g5):
        """u v t p rho ri, F1..F5, G1..G5"""
        c2, c3 = rho * u, rho * v
        return torch.stack([u, v, t, p, rho, ri, c2, c2 * u + p, c2 * v, (c4 + p) * u, f5,
                            c3, c2 * v, c3 * v + p, (c4 + p) * v, g5])

    def primitives(self, c):
        """The field set of the cells and their ghosts, [16, ni+2, nj+2]."""
        f = self.flow
        rho = c[0]
        u, v = c[1] / rho, c[2] / rho
        t = (c[3] / rho - 0.5 * (u * u + v * v)) / self.cv
        w = self._set(u, v, t, rho * self.rr * t, rho, c[3], c[4] / rho, c[4] * u, c[4] * v)
        flat = w.reshape(16, -1)
        pr, op = flat[:, self.g_par], flat[:4, self.g_opp]
        pu, pv, pt, pp, prho, pri, pf5, pg5 = (pr[k] for k in (0, 1, 2, 3, 4, 5, 10, 15))
        tot = lambda rho, t, u, v: rho * (self.cv * t + 0.5 * (u * u + v * v))
        out = torch.zeros_like(pr)
        for ty in sorted(self.types):
            if ty == 2:
                gu, gv = pu.abs(), -pv
                gt = f.t0 - 0.5 * (gu * gu + gv * gv) / self.cp
                gr = (self.s0 / (self.rr * gt)) ** (1.0 / (1.0 - f.gama))
                mu = self.amu(gt)
                g = self._set(gu, gv, gt, gr * self.rr * gt, gr, tot(gr, gt, gu, gv), mu / gr, mu * gu, mu * gv)
            elif ty == 3:
                gu, gv, gt = (2.0 * pu - op[0]).abs(), 2.0 * pv - op[1], 2.0 * pt - op[2]
                gp = torch.full_like(pp, f.pamb) if f.pamb >= 0.0 else 2.0 * pp - op[3]
                gr = gp / (self.rr * gt)
                g = self._set(gu, gv, gt, gp, gr, tot(gr, gt, gu, gv), prho * pri / gr, pf5, pg5)
            elif ty == 4:
                g = self._set(pu, -pv, pt, pp, prho, tot(prho, pt, pu, pv), pri, pf5, -pg5)
            elif ty == 5:
                g = torch.cat([torch.stack([-pu, -pv, pt, pp, prho, -pri, -pr[6], 2.0 * pp - pr[7], -pr[8], -pr[9],
                                            -pf5, -pr[11], -pr[12], 2.0 * pp - pr[13], -pr[14], -pg5])])
            elif ty == 6:
                g = self._port(c, pu, pv, pp, prho, tot)
            else:
                raise NotImplementedError(ty)
            out = torch.where(self.g_type == ty, g, out)
        full = torch.zeros((16, (self.ni + 2) * (self.nj + 2)), dtype=F64, device=c.device)
        full = full.index_copy(1, self.g_pad, out).reshape(16, self.ni + 2, self.nj + 2)
        return torch.nn.functional.pad(w, (1, 1, 1, 1)) + full

    def _port(self, c, pu, pv, pp, prho, tot):
        """Type 6: mass injection, erosive where the port flux is strong."""
        f = self.flow
        six = self.g_type == 6
        ones = torch.ones_like(pu)
        flux = c[1] * (self.yc[self.inner] if f.iaxis == 1 else 1.0)
        (_, y1, _, y2), (_, y3, _, y4) = self.faces[0], self.faces[2]
        dj, di = 0.5 * ((y3 + y4) - (y1 + y2)), 0.5 * ((y2 + y3) - (y1 + y4))
        gport = torch.cat([-(flux * dj).sum(1), (flux * di).sum(0), (flux * dj).sum(1), -(flux * di).sum(0)])
        at = [(slice(None), 0), (-1, slice(None)), (slice(None), -1), (0, slice(None))]
        sx = torch.where(six, torch.cat([self.sx[k][at[k]] for k in range(4)]), ones)
        sy = torch.where(six, torch.cat([self.sy[k][at[k]] for k in range(4)]), ones)
        ycg = self.yc.reshape(-1)[self.g_pad]
        ycp = self.yc[self.inner].reshape(-1)[self.g_par]
        dnr = torch.sqrt(sx * sx + sy * sy)
        enx, eny = -sx / dnr, -sy / dnr
        dh = torch.where(six, (ycg + ycp).abs(), ones)
        gp = torch.where(six, 2.0 * gport / (dh * dh) if f.iaxis == 1 else gport / dh, ones)
        rdot = f.acomb * (pp / 98066.5) ** f.ancomb * torch.where(six, self.g_inj, ones)

        def state(rate):
            vel = f.rhoprop / prho * rate
            u, v = 2.0 * vel * enx - pu, 2.0 * vel * eny - pv
            return u, v, f.tflame - 0.5 * (u * u + v * v) / self.cp

        t1 = state(rdot)[2]
        val = (gp / (f.rhoprop * rdot)) * (f.rhoprop * rdot * dh / self.amu(t1)) ** -0.125
        strong = val > 35.0
        eb = torch.where(strong, rdot * (1.0 + 0.023 * (torch.where(strong, val, 35.0 * ones) ** 0.8 - 35.0 ** 0.8)),
                         rdot)
        u, v, t = state(eb)
        rho = pp / (self.rr * t)
        mu = self.amu(t)
        return self._set(u, v, t, pp, rho, tot(rho, t, u, v), mu / rho, mu * u, mu * v)

    def time_step(self, c):
        u, v = c[1] / c[0], c[2] / c[0]
        t = (c[3] / c[0] - 0.5 * (u * u + v * v)) / self.cv
        dt = self.flow.cfl * self.dl / (_sqrt(u * u + v * v) + torch.sqrt(self.flow.gama * self.rr * t))
        if self.flow.local == 0:
            dt = torch.zeros_like(dt) + dt.min().clamp(max=1.0e5)
        return dt, c[0] * self.rr * t

    def dissipation(self, c, p, dt):
        def sensor(a, low=None):
            n = _around(_replicate(a))
            num = sum((v - a).abs() for v in n)
            den = sum((v + a).abs() for v in n)
            return num / (den if low is None else _dmax(den, low))

        sens = [sensor(p)] * 4 + [sensor(c[4], 8.0 * c[0] * self.rtol)]
        vd = self.vol / dt
        vn = _around(_replicate(vd))
        out = []
        for m in range(5):
            cn = _around(_replicate(c[m]))
            lap = cn[0] + cn[1] + cn[2] + cn[3] - 4.0 * c[m]
            ln, sn = _around(_replicate(lap)), _around(_replicate(sens[m]))
            d = 0.0
            for k in range(4):
                e2 = 0.25 * _dmax(sens[m], sn[k])
                e4 = _dmax(torch.zeros_like(e2), 0.00390625 - e2)
                d = d + 0.5 * (vd + vn[k]) * (e2 * (cn[k] - c[m]) - e4 * (ln[k] - lap))
            out.append(d)
        return out

    def viscous(self, w):
        f = self.flow
        val = torch.stack([w[0], w[1], w[2], w[4], w[5]])  # u v t rho ri
        node = self._four(val * self.is_cell).reshape(5, -1)
        g = val.reshape(5, -1)[:, self.g_pad]
        b = node[:, self.b_node]
        for q in self.b_g:
            b = b + g[:, q]
            ty = self.g_type[q]
            wall, flat = ty == 5, (ty == 4) | (ty == 5)
            z = torch.zeros_like(b[0])
            b = torch.stack([torch.where(wall, z, b[0]), torch.where(flat, z, b[1]), b[2], b[3],
                             torch.where(wall, z + self.rtol * f.rtred, b[4])])
        node = node.index_copy(1, self.b_node, b).reshape(5, self.ni + 1, self.nj + 1) / self.count
        node = torch.cat([node[:4], _dmax(torch.zeros_like(node[4:]) + self.rtol, node[4:])])
        corner = [node[:, :-1, :-1], node[:, 1:, :-1], node[:, 1:, 1:], node[:, :-1, 1:]]
        A, C = val[:, 1:-1, 1:-1], _around(val)
        xa, ya, xn, yn = self.xc[self.inner], self.yc[self.inner], _around(self.xc), _around(self.yc)
        vis = 0.0
        for k in range(4):
            xb, yb, xd, yd = self.faces[k]
            B, D = corner[k], corner[(k + 1) % 4]
            det = (xa - xn[k]) * (yb - yd) - (xb - xd) * (ya - yn[k])
            gx = ((A - C[k]) * (yb - yd) - (B - D) * (ya - yn[k])) / det
            gy = ((B - D) * (xa - xn[k]) - (A - C[k]) * (xb - xd)) / det
            u, v, t, rho, r = 0.25 * (A + B + C[k] + D)
            div = gx[0] + gy[1]
            if f.iaxis == 1:
                ym = 0.5 * (yb + yd)
                near = ym < 0.001
                div = div + torch.where(near, gy[1], v / torch.where(near, torch.ones_like(ym), ym))
            mu = self.amu(t)
            chi = rho * r / (mu * CMU)
            mut = rho * r * torch.tanh(ALPHA_T * chi * chi) / torch.tanh(BETA_T * chi * chi)
            eff, cond = mu + mut, mu * self.cp / f.prandtl + mut * self.cp / f.prandtlt
            txx, tyy = eff * (2.0 * gx[0] - 2.0 / 3.0 * div), eff * (2.0 * gy[1] - 2.0 / 3.0 * div)
            txy = eff * (gy[0] + gx[1])
            sx, sy = self.sx[k], self.sy[k]
            vis = vis + torch.stack([txx * sx + txy * sy, txy * sx + tyy * sy,
                                     (u * txx + v * txy + cond * gx[2]) * sx + (u * txy + v * tyy + cond * gy[2]) * sy,
                                     eff * (gx[4] * sx + gy[4] * sy)])
        return vis

    def sources(self, w):
        f = self.flow
        val = torch.stack([_sqrt(w[0] * w[0] + w[1] * w[1]), w[5], w[0], w[1]])  # |V| ri u v
        F, X, Y = _around(val), _around(self.xc), _around(self.yc)
        det = (X[0] - X[2]) * (Y[1] - Y[3]) - (X[1] - X[3]) * (Y[0] - Y[2])
        gx = ((F[0] - F[2]) * (Y[1] - Y[3]) - (F[1] - F[3]) * (Y[0] - Y[2])) / det
        gy = ((F[1] - F[3]) * (X[0] - X[2]) - (F[0] - F[2]) * (X[1] - X[3])) / det
        u, v, t, p, rho, ri = (w[k][self.inner] for k in range(6))
        mu = self.amu(t)
        chi = rho * ri / (CMU * mu)
        fmu = torch.tanh(ALPHA_T * chi * chi) / torch.tanh(BETA_T * chi * chi)
        fr2 = torch.tanh(torch.sqrt(chi)) / torch.tanh(chi * math.sqrt(2.0 * math.sqrt(CMU)))
        mut = fmu * rho * ri
        dee = torch.where(gx[0] * gx[1] + gy[0] * gy[1] > 0.0, gx[1] ** 2 + gy[1] ** 2, torch.zeros_like(mu))
        div, sq = gx[2] + gy[3], 2.0 * (gx[2] ** 2 + gy[3] ** 2) + (gy[2] + gx[3]) ** 2
        s3 = None
        if f.iaxis == 1:
            yc = self.yc[self.inner]
            near = yc < 0.001
            vy = torch.where(near, gy[3], v / torch.where(near, torch.ones_like(yc), yc))
            div, sq = div + vy, sq + 2.0 * vy ** 2
            s3 = (p - (mu + mut) * (2.0 * vy - 2.0 / 3.0 * div)) / yc
        pk = mut / rho * (sq - 2.0 / 3.0 * div ** 2)
        pk = _dmax(pk, torch.zeros_like(pk))
        pw = (mut / _dmax(mut, 0.001 * mu)) ** f.npseudo
        return s3, (rho * (21.479 - 21.394 * fr2) * _sqrt(ri * pk) - rho * 1.5 * dee) * pw

    def iteration(self, old):
        """Q_old [5, ni, nj] -> Q_new."""
        dt, p = self.time_step(old)
        d = self.dissipation(old, p, dt)
        c, vis = old, None
        for alpha in ALPHA_RK:
            w = self.primitives(c)
            if vis is None:
                vis = self.viscous(w)
            s3, s5 = self.sources(w)
            F, G = w[6:11], w[11:16]
            Fi, Gi, Fn, Gn = F[:, 1:-1, 1:-1], G[:, 1:-1, 1:-1], _around(F), _around(G)
            R = 0.5 * sum((Fi + Fn[k]) * self.sx[k] + (Gi + Gn[k]) * self.sy[k] for k in range(4))
            R = list(R)
            if s3 is not None:
                R[2] = R[2] - self.vol * s3
            R[4] = R[4] - self.vol * s5
            k = alpha * dt / self.vol
            new = [old[0] - k * (R[0] - d[0])]
            new += [old[m] - k * (0.5 if m == 4 else 1.0) * (R[m] - vis[m - 1] - d[m]) for m in range(1, 5)]
            new[4] = new[0] * _dmax(torch.zeros_like(new[0]) + self.rtol, new[4] / new[0])
            c = torch.stack(new)
        return c


def _advance(mesh, flow, q, n):
    """Q after n iterations and the residual record of the last."""
    sch = _Scheme(mesh, flow, formats.rinit_cold(flow))
    q = q.reshape(5, sch.ni, sch.nj)
    with torch.no_grad():
        for _ in range(n):
            old, q = q, sch.iteration(q)
        rec = (old - q).abs().reshape(5, -1).amax(1)
        floor = torch.tensor([1.0e-10] * 4 + [1.0e-20], dtype=F64, device=q.device)
        return q.reshape(5, -1).contiguous(), torch.maximum(rec, floor)


def exact(case, seed):
    kind = case["kind"]
    if kind == "time_step":
        st = prepare(case, seed)
        flow, q = meshes.ramp_flow(), st["q"]
        rr = 8314.0 / flow.amol
        u, v = q[1] / q[0], q[2] / q[0]
        t = (q[3] / q[0] - 0.5 * (u * u + v * v)) / (rr / (flow.gama - 1.0))
        dt = st["cfldl"] / (torch.sqrt(u * u + v * v) + torch.sqrt(flow.gama * rr * t))
        return dt, dt.min().clamp(max=1.0e5).reshape(1)
    if kind == "batch":
        outs, recs = [], []
        for k, c in enumerate(_sweep(case)):
            mesh, flow = c.mesh(), c.flow()
            q, rec = _advance(mesh, flow, _state(flow, c.nx, c.ny, seed * 100 + k), case["iters"])
            outs.append(q.cpu())
            recs.append(rec.cpu().numpy()[None])
        return outs if case["precision"] else (outs, np.concatenate(recs))
    mesh, flow = _setup(case["family"], case["ni"], case["nj"], case["local"])
    q = _state(flow, case["ni"], case["nj"], seed)
    if kind in ("solve", "coupled", "general"):
        out, rec = _advance(mesh, flow, q, case["iters"])
        if kind == "solve":
            return out
        if kind == "coupled":
            return out.cpu() if case["precision"] else (out.cpu(), rec.cpu())
        perm = meshes.renumbered_mesh(mesh, seed=3)[1]
        host = np.empty(tuple(out.shape))
        host[:, perm] = out.cpu().numpy()
        return host if case["precision"] else (host, rec.cpu().numpy()[None])
    # the reverse of each iteration by automatic differentiation
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 11)
    seed_lam = torch.randn(q.shape, generator=g, device="cuda", dtype=F64) / q.abs().amax(dim=1, keepdim=True)
    sch = _Scheme(mesh, flow, formats.rinit_cold(flow))
    shape = (5, sch.ni, sch.nj)
    states = [q.reshape(shape)]
    with torch.no_grad():
        for _ in range(case["iters"] if case["mode"] == "transient" else 0):
            states.append(sch.iteration(states[-1]))
    lam = seed_lam.reshape(shape)
    for k in range(case["iters"] - 1, -1, -1):
        at = (states[k] if case["mode"] == "transient" else states[0]).clone().requires_grad_(True)
        (lam,) = torch.autograd.grad(sch.iteration(at), [at], grad_outputs=lam)
        if case["mode"] == "fixed":
            lam = lam + seed_lam.reshape(shape)
    lam = lam.reshape(5, -1)
    return (lam, states[-1].reshape(5, -1), None) if case["mode"] == "transient" else lam
