"""Timing cases of the explicit time step: the calls a user's program makes.

A case is a mesh of one of the package's generators, a scheme, a precision and
an entry point:

  residual   one evaluation of the cell residuals of a state on the device
             (lfm_solver_residual_noalloc): the smallest call there is
  advance    host state in, a number of time steps, host state out
             (Solver.advance between page-locked arrays): what lies between
             two outputs of a run
  monitored  the loop of a run with adjustTimeStep, averages and probes: per
             step the CFL number, the next time step, one step, the pressure
             sums and the probes
  batch      many uneven cases advanced together (Batch.advance)
  serve      solve requests of different meshes and lengths submitted to a
             server and collected (Server.submit / wait / result)

``exact`` restates the schemes in 64-bit torch from the polyMesh alone.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from lfm_public_gb300 import _native as N
from lfm_public_gb300 import cases as G

M1, M2, AUSM = 0, 1, 2
PRECISION = {"fp64": N.LFM_FP64, "fp32_bulk": N.LFM_FP32_BULK}
STAGES = 5
MAX_CO = 0.1       # of the monitored runs
SPINE = 9          # probes of the monitored runs


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # a host program that drives its own time integration asks for one
        # residual at a time on a small mesh: launches and latency
        {"name": "residual_cyl96x64_m2_fp64", "kind": "residual", "mesh": "cylinder", "a": 96, "b": 64, "c": 1,
         "scheme": M2, "precision": "fp64", "steps": 1},
        # a first trial on a coarse grid
        {"name": "vortex48_m1_fp64", "kind": "advance", "mesh": "vortex", "a": 48, "b": 48, "c": 1,
         "scheme": M1, "precision": "fp64", "steps": 40},
        # the 256 x 256 isentropic vortex, inviscid, in both precisions
        {"name": "vortex256_m1_fp64", "kind": "advance", "mesh": "vortex", "a": 256, "b": 256, "c": 1,
         "scheme": M1, "precision": "fp64", "steps": 20},
        {"name": "vortex256_m1_fp32", "kind": "advance", "mesh": "vortex", "a": 256, "b": 256, "c": 1,
         "scheme": M1, "precision": "fp32_bulk", "steps": 40},
        # the headline mesh: 768 x 512 cylinder O-grid, viscous, both precisions
        {"name": "cyl768x512_m1_fp64", "kind": "advance", "mesh": "cylinder", "a": 768, "b": 512, "c": 1,
         "scheme": M1, "precision": "fp64", "steps": 10},
        {"name": "cyl768x512_m1_fp32", "kind": "advance", "mesh": "cylinder", "a": 768, "b": 512, "c": 1,
         "scheme": M1, "precision": "fp32_bulk", "steps": 20},
        # the shock-capturing scheme with limited reconstruction, odd sizes
        {"name": "cyl331x217_ausm_fp32", "kind": "advance", "mesh": "cylinder", "a": 331, "b": 217, "c": 1,
         "scheme": AUSM, "precision": "fp32_bulk", "steps": 20},
        # a 3D wake section in the reference's arithmetic, odd sizes
        {"name": "wake97x61x23_m2_fp64", "kind": "advance", "mesh": "wake", "a": 97, "b": 61, "c": 23,
         "scheme": M2, "precision": "fp64", "steps": 10},
        # the largest: a 3D wake whose working set (0.9 GB) is far beyond L2
        {"name": "wake192x128x48_m2_fp32", "kind": "advance", "mesh": "wake", "a": 192, "b": 128, "c": 48,
         "scheme": M2, "precision": "fp32_bulk", "steps": 10},
        # a run that adapts its time step and keeps averages and probes
        {"name": "monitored_cyl257x131_m2_fp64", "kind": "monitored", "mesh": "cylinder", "a": 257, "b": 131, "c": 1,
         "scheme": M2, "precision": "fp64", "steps": 12},
        # a parameter sweep: quads and triangulations, 8k-120k cells
        {"name": "batch8", "kind": "batch", "count": 8, "cells_min": 8000, "cells_max": 120000, "mix": 1, "steps": 20},
        # a burst of requests of different sizes, the large ones on their own solvers
        {"name": "serve6", "kind": "serve", "count": 6, "cells_min": 10000, "cells_max": 150000, "mix": 2,
         "steps": 100},
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["advance"] * 6 + ["residual", "monitored", "batch", "serve"])
    if kind in ("batch", "serve"):
        lo = _between(rng, 4000, 16000)
        return {"kind": kind, "count": rng.randint(3, 8), "cells_min": lo, "cells_max": lo * rng.randint(2, 8),
                "mix": rng.randint(1, 1 << 20),
                "steps": rng.randint(10, 20) if kind == "batch" else rng.randint(50, 100)}
    precision = rng.choice(["fp64", "fp32_bulk"])
    mesh = rng.choice(["vortex", "cylinder", "tri", "wake"])
    if kind in ("residual", "monitored"):
        mesh = "cylinder"
    if mesh == "vortex":
        a = _between(rng, 40, 600)
        return {"kind": kind, "mesh": mesh, "a": a, "b": max(32, int(a * rng.uniform(0.5, 1.5))), "c": 1,
                "scheme": rng.choice([M1, M2]), "precision": precision, "steps": rng.randint(10, 20)}
    if mesh == "tri":
        return {"kind": kind, "mesh": mesh, "a": _between(rng, 40, 400), "b": 1, "c": 1,
                "scheme": rng.choice([M1, M2]), "precision": precision, "steps": rng.randint(10, 20)}
    if mesh == "wake":
        a = _between(rng, 36, 150)
        return {"kind": kind, "mesh": mesh, "a": a, "b": max(16, int(a * rng.uniform(0.5, 0.8))),
                "c": max(4, int(a * rng.uniform(0.1, 0.3))), "scheme": rng.choice([M1, M2, AUSM]),
                "precision": precision, "steps": rng.randint(3, 8)}
    # a residual's scratch holds up to about 120k 2D cells in FP64
    b = _between(rng, 24, 180) if kind == "residual" else _between(rng, 32, 500)
    return {"kind": kind, "mesh": mesh, "a": int(b * rng.uniform(1.2, 1.6)), "b": b, "c": 1,
            "scheme": rng.choice([M1, M2, AUSM]), "precision": precision,
            "steps": 1 if kind == "residual" else rng.randint(8, 16)}


# ---------------------------------------------------------------------------
# what a program has in hand
# ---------------------------------------------------------------------------
def _mesh_case(case):
    if case["mesh"] == "vortex":
        return G.vortex_case(n=case["a"], ny=case["b"], solver=case["scheme"])
    if case["mesh"] == "tri":
        return G.tri_case(n=case["a"], seed=case["a"], mach=0.3, beta=3.0, solver=case["scheme"])
    if case["mesh"] == "cylinder":
        return G.cylinder_case(n_theta=case["a"], n_r=case["b"], solver=case["scheme"], minmod=True)
    return G.cylinder_case(n_theta=case["a"], n_r=case["b"], n_span=case["c"], solver=case["scheme"], reynolds=3900.0,
                           minmod=case["scheme"] == AUSM)


@functools.lru_cache(maxsize=3)
def _described(key):
    """A mesh and its solver description. A program that runs several initial
    states on one mesh reads the mesh once."""
    c = _mesh_case(dict(key))
    return c, N.CaseHandle.from_case(c)


def _described_of(case):
    return _described(tuple((k, case[k]) for k in ("mesh", "a", "b", "c", "scheme")))


def _noisy(q, dim, u_inf, rng):
    """The state q with uniform noise of +-1% of the free-stream speed on each
    velocity component (the start of the 3D wake runs)."""
    q = q.copy()
    u = q[1:1 + dim] / q[0]
    v = u + rng.uniform(-0.01, 0.01, size=u.shape) * u_inf
    q[1 + dim] += 0.5 * q[0] * (np.sum(v * v, axis=0) - np.sum(u * u, axis=0))
    q[1:1 + dim] = q[0] * v
    return q


def _state(q0, c, seed, k=0):
    u_inf = math.sqrt(sum(x * x for x in c.U_inf))
    return _noisy(q0, c.dim, u_inf, np.random.default_rng([int(seed), k]))


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def _pinned_copy(q):
    out = _pinned(q.shape)
    out[...] = q
    return out


def _sweep(case, seed):
    """The meshes of a batch or of a burst of requests: vortices on quads and
    triangulations and, among the requests, cylinder O-grids and wakes."""
    rng = np.random.default_rng(case["mix"])
    out = []
    for k in range(case["count"]):
        cells = math.exp(rng.uniform(math.log(case["cells_min"]), math.log(case["cells_max"])))
        mach, beta, scheme = float(rng.uniform(0.1, 0.6)), float(rng.uniform(1, 4)), int(rng.integers(0, 2))
        shape = k % 2 if case["kind"] == "batch" else k % 4
        if shape == 0:
            c = G.vortex_case(n=int(math.sqrt(cells)), mach=mach, beta=beta, solver=scheme)
        elif shape == 1:
            c = G.tri_case(n=int(math.sqrt(cells / 2)), seed=case["mix"] + k, mach=mach, beta=beta, solver=scheme)
        elif shape == 2:
            nr = int(math.sqrt(cells / 1.5))
            c = G.cylinder_case(n_theta=int(1.5 * nr), n_r=nr, solver=scheme, minmod=True)
        else:
            s = (cells / (384 * 256 * 96)) ** (1.0 / 3.0)
            c = G.cylinder_case(n_theta=int(384 * s), n_r=int(256 * s), n_span=max(4, int(96 * s)), solver=M2,
                                reynolds=3900.0, minmod=False)
        r = np.random.default_rng([int(seed), k])
        u_inf = math.sqrt(sum(x * x for x in c.U_inf))
        c.fields["U"][:, :c.dim] += r.uniform(-0.01, 0.01, size=(c.n_cells, c.dim)) * u_inf
        out.append(c)
    return out


def _requests(case, seed):
    """(mesh, steps) of a burst: every request has its own length."""
    rng = np.random.default_rng(case["mix"] + 1)
    return [(c, int(case["steps"] * rng.uniform(0.5, 1.0))) for c in _sweep(case, seed)]


def prepare(case, seed):
    st = {"case": case}
    if case["kind"] == "batch":
        st["meshes"] = _sweep(case, seed)
        handles = [N.CaseHandle.from_case(c) for c in st["meshes"]]
        b = N.Batch(arena_bytes=sum(N.Batch.case_bytes(h) for h in handles) + (16 << 20), max_cases=len(handles))
        st["slots"] = [b.add(h, c.delta_t) for h, c in zip(handles, st["meshes"])]
        st["q_in"] = [_pinned_copy(h.q0()) for h in handles]
        st["q_out"] = [_pinned(q.shape) for q in st["q_in"]]
        st["batch"] = b
        return st
    if case["kind"] == "serve":
        st["requests"] = [(N.CaseHandle.from_case(c), c.delta_t, n) for c, n in _requests(case, seed)]
        st["server"] = N.Server(arena_bytes=1 << 30, chunk_steps=50, solo_cells=30000, max_solo=2)
        return st
    c, ch = _described_of(case)
    q = _state(ch.q0(), c, seed)
    st["dt"] = c.delta_t
    s = st["solver"] = N.Solver(ch, precision=PRECISION[case["precision"]])
    if case["kind"] == "residual":
        st["q"] = torch.from_numpy(q).cuda()
        st["res"] = torch.empty_like(st["q"])
        N.check(N.load_library().lfm_solver_residual_noalloc(s._h, st["q"].data_ptr(), ch.desc.n_cells,
                                                             st["res"].data_ptr(), None))
        return st
    st["q_in"], st["q_out"] = _pinned_copy(q), _pinned(q.shape)
    if case["kind"] == "monitored":
        st["probes"] = np.linspace(0, ch.desc.n_cells - 1, SPINE).astype(np.int64)
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(st):
    case = st["case"]
    if case["kind"] == "advance":
        return st["solver"].advance(st["q_in"], case["steps"], st["dt"], st["q_out"])
    if case["kind"] == "residual":
        q, res = st["q"], st["res"]
        N.check(N.load_library().lfm_solver_residual_noalloc(
            st["solver"]._h, q.data_ptr(), q.shape[1], res.data_ptr(),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return res
    if case["kind"] == "batch":
        st["batch"].advance(st["slots"], st["q_in"], case["steps"], st["q_out"])
        return st["q_out"]
    if case["kind"] == "serve":
        srv = st["server"]
        ids = [srv.submit(h, dt, n) for h, dt, n in st["requests"]]
        out = []
        for i in ids:
            srv.wait(i)
            out.append(srv.result(i)[0])
        return out
    s = st["solver"]
    s.set_state(st["q_in"])
    s.stats_reset()
    s.probes_set(st["probes"], case["steps"])
    log = np.empty((case["steps"], 2))
    for k in range(case["steps"]):
        dt = s.min_dt(MAX_CO)
        log[k] = dt, s.cfl(dt)
        s.step(1, dt)
        s.stats_accumulate(k + 1)
        s.probes_record()
    s.sync()
    p_avg, p_rms = s.stats_get(case["steps"])
    return {"q": s.get_state(st["q_out"]), "log": log, "p_avg": p_avg, "p_rms": p_rms, "probes": s.probes_read()}


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------
def _cell_work(dim, faces_per_cell, scheme, viscous):
    """(bytes, flops per stage) of a cell: its state in and out once and the
    mesh read once (per face two cell labels, S, K, the weight and the
    Laplacian constant; per cell 1/V and the sponge), in FP64; the flops of
    its share of the faces, of its gradients and of its update."""
    nq, f = dim + 2, faces_per_cell / 2
    face = {M1: 9 + 13 * dim, M2: 16 + 11 * dim, AUSM: 150 + 60 * dim}[scheme]
    cell = faces_per_cell * nq + 9 * nq
    if viscous:
        face += 3 * (dim * dim + 2 * dim) + 2 * dim * (dim + 3) + 6
        cell += faces_per_cell * 2 * (dim * dim + dim) + 4 * dim * dim
    if scheme == AUSM:
        cell += faces_per_cell * 2 * (dim * dim + 2 * dim)
    return 16 * nq + 16 + f * (8 + 8 * (2 * dim + 2)), f * face + cell


def _case_sizes(case):
    """(cells, dim, faces per cell, scheme, viscous, steps) of each mesh."""
    if case["kind"] in ("batch", "serve"):
        pairs = _requests(case, 0) if case["kind"] == "serve" else [(c, case["steps"]) for c in _sweep(case, 0)]
        return [(c.n_cells, c.dim, 6 if c.dim == 3 else 3 if c.name.startswith("tri") else 4, c.solver, c.mu > 0, n)
                for c, n in pairs]
    a, b = case["a"], case["b"]
    if case["mesh"] == "tri":
        return [(2 * a * a, 2, 3, case["scheme"], False, case["steps"])]
    dim = 3 if case["mesh"] == "wake" else 2
    return [(a * b * case["c"], dim, 2 * dim, case["scheme"], case["mesh"] != "vortex", case["steps"])]


def work(case):
    total = {"bytes": 0.0, "flops": 0.0}
    for cells, dim, faces, scheme, viscous, steps in _case_sizes(case):
        by, fl = _cell_work(dim, faces, scheme, viscous)
        total["bytes"] += by * cells
        total["flops"] += fl * cells * (1 if case["kind"] == "residual" else STAGES * steps)
    return total


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
RK_A = (0.0, -0.4178904745, -1.192151694643, -1.697784692471, -1.514183444257)
RK_B = (0.1496590219993, 0.3792103129999, 0.8229550293869, 0.6994504559488, 0.1530572479681)


class _Plain:
    """A polyMesh case in 64-bit torch: geometry, boundary states and the
    schemes, face by face, sums by index_add."""

    def __init__(self, c):
        dev = self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.c, D = c, c.dim
        self.D, self.nc = D, c.n_cells
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
        pts, offs, fp = t(c.points), t(c.face_offsets), t(c.face_points)
        own, nei = t(c.owner), t(c.neighbour)
        nf, ni = len(own), len(nei)
        # faces: a triangle's own centre and area, larger faces as a fan about
        # the average of their points
        ctr, area = torch.zeros(2, nf, 3, dtype=torch.float64, device=dev).unbind(0)
        on_boundary = torch.zeros(len(pts), dtype=torch.bool, device=dev)
        sizes = offs[1:] - offs[:-1]
        for n in sizes.unique().tolist():
            f = torch.nonzero(sizes == n)[:, 0]
            P = pts[fp[offs[f][:, None] + torch.arange(n, device=dev)]]
            if n == 3:
                ctr[f] = P.mean(1)
                area[f] = 0.5 * torch.linalg.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0])
                continue
            mid = P.mean(1, keepdim=True)
            nxt = P.roll(-1, 1)
            cr = torch.linalg.cross(nxt - P, mid - P)
            a = cr.norm(dim=2, keepdim=True)
            ctr[f] = ((P + nxt + mid) * a).sum(1) / (3 * a.sum(1))
            area[f] = 0.5 * cr.sum(1)
        # cells: pyramids from the faces to the average face centre
        est = self._sum(own, ctr) + self._sum(nei, ctr[:ni])
        cnt = self._sum(own, torch.ones_like(ctr)) + self._sum(nei, torch.ones_like(ctr[:ni]))
        est = est / cnt
        vol, cen = 0.0, 0.0
        for cell, s, n in ((own, 1.0, nf), (nei, -1.0, ni)):
            p3 = s * (area[:n] * (ctr[:n] - est[cell])).sum(1, keepdim=True)
            vol = vol + self._sum(cell, p3)
            cen = cen + self._sum(cell, p3 * (0.75 * ctr[:n] + 0.25 * est[cell]))
        cen = cen / vol
        self.vol = vol[:, 0] / 3
        # solver order: the cells that touch a point of a boundary patch come first
        face_pt = torch.repeat_interleave(torch.arange(nf, device=dev), sizes)
        for p in c.patches:
            if p.type != "empty":
                on_boundary[fp[offs[p.start]:offs[p.start + p.size]]] = True
        touched = torch.zeros(nf, dtype=torch.bool, device=dev)
        touched[face_pt[on_boundary[fp]]] = True
        first = torch.zeros(self.nc, dtype=torch.bool, device=dev)
        first[own[touched]] = True
        first[nei[touched[:ni]]] = True
        self.order = torch.cat([torch.nonzero(first)[:, 0], torch.nonzero(~first)[:, 0]])
        # faces between cells, then one ghost per boundary face
        P, Q, S, d, xf = [own[:ni]], [nei], [area[:ni]], [cen[nei] - cen[own[:ni]]], [ctr[:ni]]
        gkind, gP, gS, gx = [], [], [], []
        start = {p.name: p.start for p in c.patches}
        for p in c.patches:
            f = torch.arange(p.start, p.start + p.size, device=dev)
            if p.type == "cyclic":
                o = f - p.start + start[p.neighbour]
                if start[p.neighbour] > p.start:
                    P.append(own[f]), Q.append(own[o]), S.append(area[f]), xf.append(ctr[f])
                    d.append(cen[own[o]] - cen[own[f]] + ctr[f] - ctr[o])
            elif p.type != "empty":
                kind = 1 if p.type == "wall" else {"inlet": 2, "outlet": 3}[p.name]
                gkind.append(torch.full((p.size,), kind, device=dev))
                gP.append(own[f]), gS.append(area[f]), gx.append(ctr[f])
        self.P, self.S = torch.cat(P + gP), torch.cat(S + gS)[:, :D]
        self.ni = sum(len(x) for x in Q)
        self.gkind, self.gP = torch.cat(gkind), torch.cat(gP)
        self.Q = torch.cat(Q + [self.nc + torch.arange(len(self.gP), device=dev)])
        dP = (cen[self.P] - torch.cat(xf + gx))[:, :D]
        gs = self.S[self.ni:]
        gd = 2 * (dP[self.ni:] * gs).sum(1, keepdim=True).abs() * gs / (gs * gs).sum(1, keepdim=True)
        self.d = torch.cat([torch.cat(d)[:, :D], gd])
        dN = dP + self.d
        self.w = ((self.S * dN).sum(1) / ((self.S * dN).sum(1) - (self.S * dP).sum(1)))
        s2 = (self.S * self.S).sum(1)
        delta = self.d * (s2 / (self.S * self.d).sum(1))[:, None]
        self.dinv = 1 / self.d.norm(dim=1)
        self.lap = delta.norm(dim=1) * self.dinv
        self.K = self.S - delta
        self.S, self.d, self.K = self.S.T.contiguous(), self.d.T.contiguous(), self.K.T.contiguous()
        # gas, sponge
        self.g, self.R = c.gamma, c.Rgas
        self.rho = c.p_inf / (self.R * c.T_inf)
        self.U = [float(c.U_inf[k]) for k in range(D)]
        u2 = sum(x * x for x in self.U)
        self.q_inf = [self.rho] + [self.rho * x for x in self.U] + [c.p_inf / (self.g - 1) + 0.5 * self.rho * u2]
        self.sponge = torch.zeros(self.nc, dtype=torch.float64, device=dev)
        if c.Ls > 0:
            x = (c.Ls - t(c.fields["alpha"])).clamp(min=0) / c.Ls
            self.sponge = 3 * (1 - c.mach * c.mach) / (c.k_sponge * c.Ls) * x * x

    def _sum(self, cell, x):
        out = torch.zeros(self.nc, x.shape[1], dtype=torch.float64, device=self.dev)
        return out.index_add_(0, cell, x)

    def from_solver(self, q):
        out = torch.empty(q.shape, dtype=torch.float64, device=self.dev)
        out[:, self.order] = torch.as_tensor(q, device=self.dev)
        return out

    def to_solver(self, q):
        return q[:, self.order]

    def pressure(self, q):
        D = self.D
        return (self.g - 1) * (q[D + 1] - 0.5 * (q[1:D + 1] ** 2).sum(0) / q[0])

    def ghosts(self, q):
        D, gm1 = self.D, self.g - 1
        qi = q[:, self.gP]
        u = qi[1:D + 1] / qi[0]
        p = gm1 * (qi[D + 1] - 0.5 * qi[0] * (u * u).sum(0))
        wall = torch.cat([qi[:1], -qi[1:D + 1], qi[D + 1:]])
        ue = torch.tensor(self.U, dtype=torch.float64, device=self.dev)[:, None]
        r = p / (self.R * self.c.T_inf)
        inlet = torch.cat([r[None], r * ue, (p / gm1 + 0.5 * r * (ue * ue).sum(0))[None]])
        r = qi[0] * self.c.p_inf / p
        outlet = torch.cat([r[None], r * u, (self.c.p_inf / gm1 + 0.5 * r * (u * u).sum(0))[None]])
        return torch.where(self.gkind == 1, wall, torch.where(self.gkind == 2, inlet, outlet))

    def gauss(self, x):
        """Gauss gradient of cell-and-ghost values x, zero on the ghosts."""
        xf = self.w * x[self.P] + (1 - self.w) * x[self.Q]
        out = torch.zeros(self.D, x.numel(), dtype=torch.float64, device=self.dev)
        out.index_add_(1, self.P, xf * self.S)
        out.index_add_(1, self.Q, -xf * self.S)
        out[:, :self.nc] /= self.vol
        out[:, self.nc:] = 0
        return out

    def minmod(self, a, b, grad, side):
        df = b - a + 1e-30
        dc = (self.d * grad).sum(0)
        sign = lambda x: torch.where(x < 0, -1.0, 1.0)  # noqa: E731
        r = torch.where(dc.abs() >= 1000 * df.abs(), 2000 * sign(dc) * sign(df) - 1, 2 * (dc / df) - 1)
        lim = r.clamp(0, 1)
        weight = lim * self.w + (1 - lim) * (1 + side) * 0.5
        return weight * a + (1 - weight) * b

    def residual(self, q):
        c, D, g, w, S, P, Q = self.c, self.D, self.g, self.w, self.S, self.P, self.Q
        qa = torch.cat([q, self.ghosts(q)], 1)
        u = qa[1:D + 1] / qa[0]
        Rp = self.pressure(qa) / qa[0]
        mix = lambda x: w * x[..., P] + (1 - w) * x[..., Q]  # noqa: E731
        mean = lambda x: 0.5 * (x[..., P] + x[..., Q])  # noqa: E731
        need = c.mu != 0 or c.solver == AUSM
        gu = torch.stack([self.gauss(u[a]) for a in range(D)]) if need else None   # [component][direction]
        if c.solver == M1:
            rho, m, R = mix(qa[0]), mix(qa[1:D + 1]), mix(Rp)
            uf = m / rho
            p, H = rho * R, g / (g - 1) * R + 0.5 * (uf * uf).sum(0)
            mS = (m * S).sum(0)
            rhs = [-mS] + [-(mS * uf[k] + p * S[k]) for k in range(D)] + [-mS * H]
        else:
            rho, m = mean(qa[0]), mean(qa[1:D + 1])
            p, H = rho * mean(Rp), mean(qa[D + 1] / qa[0] + Rp)
            if c.solver == AUSM:
                p = p + self.ausm(qa, u, Rp, gu)
            phi = (m / rho * S).sum(0)
            rhs = [-rho * phi] + [-(m[k] * phi + p * S[k]) for k in range(D)] + [-rho * H * phi]
        if c.mu != 0:
            T = Rp / self.R
            gT = self.gauss(T)
            dn, ni = self.d * self.dinv, self.ni
            gf, gTf = mix(gu), mix(gT)
            du, dT = u[:, Q] - u[:, P], T[Q] - T[P]
            gf[:, :, ni:] = (du[:, None] * dn * self.dinv)[:, :, ni:]
            gTf[:, ni:] = (dT * dn * self.dinv)[:, ni:]

            def stress(x):   # the deviatoric stress, trace taken as the scheme has it
                tau = c.mu * (x + x.transpose(0, 1))
                tr = sum(x[a, a] for a in range(D))
                for a in range(D):
                    tau[a, a] = (2.0 / 3.0) * c.mu * (3 * x[a, a] - tr)
                return tau
            sig = mix(torch.stack([(u * row).sum(0) for row in stress(gu)]))
            sig[:, ni:] = torch.stack([(mix(u) * row).sum(0) for row in stress(gf)])[:, ni:]
            tr = sum(gf[a, a] for a in range(D))
            for a in range(D):
                div = c.mu * (gf[:, a] * S).sum(0) - (2.0 / 3.0) * c.mu * tr * S[a]
                rhs[a + 1] = rhs[a + 1] + div + c.mu * (self.lap * du[a] + (self.K * gf[a]).sum(0))
            rhs[D + 1] = rhs[D + 1] + (sig * S).sum(0) + c.Cp * c.mu / c.Pr * (self.lap * dT + (self.K * gTf).sum(0))
        rhs = torch.stack(rhs)
        out = torch.zeros(D + 2, self.nc, dtype=torch.float64, device=self.dev)
        out.index_add_(1, P, rhs)
        return out.index_add_(1, Q[:self.ni], -rhs[:, :self.ni])

    def ausm(self, qa, u, Rp, gu):
        """AUSM+ pressure dissipation on limited states, scaled by a shock sensor."""
        D, P, Q, S = self.D, self.P, self.Q, self.S
        c = (self.g * Rp).sqrt()
        c = 0.5 * (c[P] + c[Q])
        div = sum(gu[a, a] for a in range(D))
        curl = sum((gu[a, b] - gu[b, a]) ** 2 for a in range(D) for b in range(a + 1, D))
        sensor = (-div / (div * div + curl + 4e-2).sqrt()).clamp(min=0)
        theta = 0.5 * (sensor[P] + sensor[Q])
        limited = lambda x, grad: (self.minmod(x[P], x[Q], grad[:, P], 1.0),  # noqa: E731
                                   self.minmod(x[P], x[Q], grad[:, Q], -1.0))
        zero = torch.zeros_like(gu[0])
        grad = self.gauss if self.c.minmod else (lambda x: zero)
        p = qa[0] * Rp
        un = [0.0, 0.0]
        for a in range(D):
            up = limited(u[a], grad(u[a]))
            un = [un[k] + up[k] * S[a] for k in (0, 1)]
        rP, rN = limited(qa[0], grad(qa[0]))
        pP, pN = limited(p, grad(p))
        norm = (S * S).sum(0)
        M2_ = (un[0] ** 2 + un[1] ** 2) / (2 * c * c * norm)
        MP, MN = un[0] / (norm.sqrt() * c), un[1] / (norm.sqrt() * c)
        M0 = M2_.clamp(0.04, 1.0).sqrt()
        fa = M0 * (2 - M0)
        al = 3 * (5 * fa * fa - 4) / 16

        def p5(M, s):
            a, b = 0.25 * (M + s) ** 2, 0.25 * (M - s) ** 2
            return torch.where(M.abs() < 1, s * a * ((2 * s - M) + 16 * al * M * b), 0.5 * (M + s * M.abs()) / M)
        half = pN * (p5(MN, 1.0) - p5(MN, -1.0)) - pP * (p5(MP, 1.0) - p5(MP, -1.0))
        pu = -0.75 * p5(MP, 1.0) * p5(MN, -1.0) * (rP + rN) * c * fa * (un[1] - un[0])
        return theta * (pu - 0.5 * half)

    def step(self, q, dt):
        dq = torch.zeros_like(q)
        inf = torch.tensor(self.q_inf, dtype=torch.float64, device=self.dev)[:, None]
        for A, B in zip(RK_A, RK_B):
            dq = A * dq + dt * (self.residual(q) / self.vol + self.sponge * (inf - q))
            q = q + B * dq
        return q

    def flows(self, q, unit):
        """Per cell the sum over its faces (ghost faces too) of |momentum . S|."""
        s = self.S / self.S.norm(dim=0) if unit else self.S
        m = q[1:self.D + 1]
        out = torch.zeros(self.nc, dtype=torch.float64, device=self.dev)
        out.index_add_(0, self.P, (m[:, self.P] * s).sum(0).abs())
        nb = self.Q[:self.ni]
        return out.index_add_(0, nb, (m[:, nb] * s[:, :self.ni]).sum(0).abs())

    def initial(self):
        f = self.c.fields
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=self.dev)  # noqa: E731
        p, T, U = t(f["p"]), t(f["T"]), t(f["U"])[:, :self.D].T
        rho = p / (self.R * T)
        return torch.cat([rho[None], rho * U, (p / (self.g - 1) + 0.5 * rho * (U * U).sum(0))[None]])


def _advanced(c, q, steps, dt):
    m = _Plain(c)
    q = m.initial() if q is None else m.from_solver(q)
    for _ in range(steps):
        q = m.step(q, dt)
    return m.to_solver(q).cpu().numpy()


def exact(case, seed):
    if case["kind"] == "batch":
        return [_advanced(c, None, case["steps"], c.delta_t) for c in _sweep(case, seed)]
    if case["kind"] == "serve":
        return [_advanced(c, None, n, c.delta_t) for c, n in _requests(case, seed)]
    c, ch = _described_of(case)
    q0 = _state(ch.q0(), c, seed)
    if case["kind"] == "advance":
        return _advanced(c, q0, case["steps"], c.delta_t)
    m = _Plain(c)
    q = m.from_solver(q0)
    if case["kind"] == "residual":
        return m.to_solver(m.residual(q))
    probes = np.linspace(0, ch.desc.n_cells - 1, SPINE).astype(np.int64)
    n, log, hist = case["steps"], [], []
    total, square = torch.zeros_like(m.vol), torch.zeros_like(m.vol)
    for k in range(n):
        dt = float((MAX_CO * q[0] * 2 * m.vol / m.flows(q, True)).min().clamp(max=100.0))
        log.append((dt, float((m.flows(q, False) / (q[0] * m.vol)).max() * dt)))
        q = m.step(q, dt)
        p = m.pressure(q)
        total += p
        square += (p - total / (k + 1)) ** 2
        hist.append((p[m.order[torch.as_tensor(probes, device=m.dev)]] - c.p_inf).cpu().numpy())
    return {"q": m.to_solver(q).cpu().numpy(), "log": np.array(log), "p_avg": (total / n)[m.order].cpu().numpy(),
            "p_rms": (square / n).sqrt()[m.order].cpu().numpy(), "probes": np.array(hist)}
