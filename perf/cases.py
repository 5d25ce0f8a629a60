"""Measured workloads of the DUGKS engine, each through the calls a user's program makes.

A case is a dict of plain values:

  kind      "steps"   FvDVM.evolution(n) and the cell fields into pinned host buffers
            "loop"    dugksFoam's time loop: per step the Courant number, dt, one step; then residuals and fields
            "batch"   Batch.step(n) over independent cavities and every case's fields
            "value", "tangent", "adjoint"   the wall objective of the gradient harness, and its derivatives
  mesh      "quads" | "triangles" | "hexes" | "channel" with n (and ny) its size
  nxi, grid velocities per direction and their rule ("nc" Newton-Cotes, "gh" half-range Gauss-Hermite)
  fp        64 (plain FP64 pipeline) or 32 (FP32 distributions, FP64 moments)
  spinup    steps the run is under way when the measured passes begin (triangles, whose time step is short
            against the relaxation time: the heat flux has to develop)

The seed gives the initial fields (a smooth flow, as mapped from another run) and the wall temperatures;
meshes depend on the sizes alone.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from dugksfoam_gb300 import cases as C
from dugksfoam_gb300 import solver

FIELDS = ("rho", "U", "T", "q")


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest: a coarse cavity on the smallest half-range Gauss-Hermite grid, where launches count
        dict(name="quads24_fp32", kind="steps", mesh="quads", n=24, nxi=8, grid="gh", kn=0.075, fp=32, steps=20),
        # the 61^2 lid-driven cavity as dugksFoam's time loop drives the solver, step by step from the host
        dict(name="loop_quads61_fp32", kind="loop", mesh="quads", n=61, nxi=28, grid="nc", kn=0.075, fp=32, steps=10),
        # the same cavity with the plain FP64 pipeline: the parity run
        dict(name="quads61_fp64", kind="steps", mesh="quads", n=61, nxi=28, grid="nc", kn=0.075, fp=64, steps=10),
        # the headline size: ~100k triangles, 32^2 velocities, Kn 0.01, FP32 distributions
        dict(name="triangles100k_fp32", kind="steps", mesh="triangles", n=224, nxi=32, grid="nc", kn=0.01, fp=32, steps=6, spinup=150),
        # the 4Z+1 velocity count that dugksFoam's own Newton-Cotes grids have: rows that are not multiples of 4
        dict(name="triangles18k_odd_fp32", kind="steps", mesh="triangles", n=95, nxi=29, grid="nc", kn=0.05, fp=32, steps=8, spinup=100),
        # plain FP64 on triangles, beside which the FP32 run is read
        dict(name="triangles24k_fp64", kind="steps", mesh="triangles", n=109, nxi=32, grid="nc", kn=0.01, fp=64, steps=3),
        # the largest: the 48^3 cubic cavity on 20^3 velocities
        dict(name="hexes48_fp32", kind="steps", mesh="hexes", n=48, nxi=20, grid="nc", kn=0.1, fp=32, steps=3),
        # 3D with the plain FP64 pipeline
        dict(name="hexes15_fp64", kind="steps", mesh="hexes", n=15, nxi=14, grid="nc", kn=0.1, fp=64, steps=3),
        # pressure-driven channel: inlet, outlet and walls (boundary types other than diffuse walls)
        dict(name="channel_fp32", kind="steps", mesh="channel", n=90, ny=45, nxi=24, grid="nc", kn=0.1, fp=32, steps=10),
        # a parameter study: seeded cavities with uneven meshes and velocity grids, advanced together
        dict(name="batch16_fp32", kind="batch", count=16, persistent=False, steps=6),
        # gradients of wall heat flux and shear by the adjoint, with checkpoints; a ragged last segment
        dict(name="adjoint_quads48", kind="adjoint", mesh="quads", n=48, nxi=28, grid="nc", kn=0.075, fp=64, steps=12, first=6, every=5),
        # the directional derivative by the tangent-linear step
        dict(name="tangent_quads32", kind="tangent", mesh="quads", n=32, nxi=28, grid="nc", kn=0.075, fp=64, steps=6, first=3, every=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["quads", "quads", "loop", "triangles", "triangles", "hexes", "channel", "batch", "gradient"])
    fp = rng.choice([32, 32, 64])
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(3, 20), persistent=rng.random() < 0.5, steps=rng.randint(3, 7))
    if kind == "gradient":
        steps = rng.randint(4, 11)
        return dict(kind=rng.choice(["value", "tangent", "adjoint"]), mesh="quads", n=rng.randint(17, 40),
                    nxi=rng.choice([26, 28, 29, 32]), grid="nc", kn=0.075, fp=64, steps=steps,
                    first=rng.randint(0, steps - 1), every=rng.randint(2, 6))
    if kind in ("quads", "loop"):
        return dict(kind="loop" if kind == "loop" else "steps", mesh="quads", n=_log(rng, 20, 150 if fp == 32 else 70),
                    nxi=rng.choice([26, 28, 29, 32, 33]), grid="nc", kn=0.075, fp=fp, steps=rng.randint(3, 10))
    if kind == "triangles":
        return dict(kind="steps", mesh="triangles", n=_log(rng, 60, 190 if fp == 32 else 95), nxi=rng.choice([28, 29, 30, 32]),
                    grid="nc", kn=0.05, fp=fp, steps=rng.randint(2, 6), spinup=120 if fp == 32 else 0)
    if kind == "hexes":
        return dict(kind="steps", mesh="hexes", n=rng.randint(9, 33 if fp == 32 else 14), nxi=rng.choice([12, 13, 14, 16, 18]),
                    grid="nc", kn=0.1, fp=fp, steps=rng.randint(2, 4))
    return dict(kind="steps", mesh="channel", n=_log(rng, 30, 140), ny=_log(rng, 15, 70), nxi=rng.choice([24, 25, 28]),
                grid="nc", kn=0.1, fp=fp, steps=rng.randint(2, 7))


# ------------------------------------------------------------------ inputs
def _triangles(n):
    """2 n^2 triangles of the unit square: an n x n grid with shifted inner nodes and one diagonal direction (flows
    on random or alternating diagonals grow without bound after some hundred steps), one cell thick, cells along a
    Morton curve, faces in OpenFOAM order, patches as the cavity's."""
    rng = np.random.default_rng(0)
    k = np.arange(n + 1)
    X, Y = (a.ravel().astype(float) for a in np.meshgrid(k, k))
    inner = (X > 0) & (X < n) & (Y > 0) & (Y < n)
    X, Y = X + inner * rng.uniform(-0.2, 0.2, X.size), Y + inner * rng.uniform(-0.2, 0.2, X.size)
    pts = np.stack([X, Y], 1) / n
    i, j = (a.ravel() for a in np.meshgrid(np.arange(n), np.arange(n)))
    a = j * (n + 1) + i
    b, c, d = a + 1, a + n + 2, a + n + 1
    tri = np.concatenate([np.stack([a, b, c], 1), np.stack([a, c, d], 1)])
    code = np.zeros(len(tri), np.int64)
    for bit in range(12):
        for ax in range(2):
            q = (pts[tri].mean(1)[:, ax] * 4095).astype(np.int64)
            code |= ((q >> bit) & 1) << (2 * bit + ax)
    tri = tri[np.argsort(code, kind="stable")]
    nT, nP = len(tri), len(pts)
    ea, eb, et = tri.ravel(), tri[:, [1, 2, 0]].ravel(), np.repeat(np.arange(nT), 3)
    key = np.minimum(ea, eb) * nP + np.maximum(ea, eb)
    order = np.argsort(key, kind="stable")  # the lower cell of an edge first
    same = key[order][1:] == key[order][:-1]
    e0, e1 = order[:-1][same], order[1:][same]
    srt = np.lexsort((et[e1], et[e0]))
    e0, e1 = e0[srt], e1[srt]
    single = np.ones(len(key), bool)
    single[np.concatenate([e0, e1])] = False
    eB = np.nonzero(single)[0]
    top = np.minimum(pts[ea[eB], 1], pts[eb[eB], 1]) > 1 - 1e-9
    edges = np.concatenate([e0, eB[top], eB[~top]])
    side = np.stack([ea[edges], eb[edges], eb[edges] + nP, ea[edges] + nP], 1)
    nI, nTop, nE = len(e0), int(top.sum()), len(edges)
    names = (("movingWall", "wall", nI, nTop), ("fixedWalls", "wall", nI + nTop, nE - nI - nTop), ("frontAndBack", "empty", nE, 2 * nT))
    return dict(
        points=np.concatenate([np.c_[pts, np.zeros(nP)], np.c_[pts, np.full(nP, 1.0 / n)]]),
        face_offsets=np.concatenate([np.arange(0, 4 * nE + 1, 4), 4 * nE + np.arange(3, 6 * nT + 1, 3)]).astype(np.int32),
        face_verts=np.concatenate([side.ravel(), tri[:, [0, 2, 1]].ravel(), (tri + nP).ravel()]).astype(np.int32),
        owner=np.concatenate([et[edges], np.arange(nT), np.arange(nT)]).astype(np.int32), neighbour=et[e1].astype(np.int32),
        n_cells=nT, patches=[dict(name=a, type=b, startFace=c, nFaces=d) for a, b, c, d in names])


@functools.lru_cache(maxsize=6)
def _mesh(mesh, n, bottom):
    if mesh == "triangles":
        return _triangles(n)
    if mesh == "hexes":
        return C.structured_mesh(n, n, n, lz=1.0, two_d=False)
    return C.structured_mesh(n, n, 1, two_d=True, bottom_patch=bottom)


def _smooth(rng, x, dims):
    """A smooth field of largest magnitude 1 at the points x."""
    f = np.zeros(len(x))
    for _ in range(4):
        k = np.zeros(3)
        k[:dims] = rng.uniform(-4 * math.pi, 4 * math.pi, dims)
        f += rng.uniform(0.5, 1.0) * np.cos(x @ k + rng.uniform(0, 2 * math.pi))
    return f / max(np.abs(f).max(), 1e-12)


@functools.lru_cache(maxsize=6)
def _centres(mesh, n, bottom):
    g = _geometry(_mesh(mesh, n, bottom))
    return g["C"], g["Cf"]


def _perturb(case, seed, centres):
    """Initial fields and wall temperatures made from the seed: temperatures within 10 %, densities within 5 %,
    velocities up to a tenth of the most probable speed (the lid moves at 0.15 of it)."""
    rng = np.random.default_rng(seed)
    x, xf = centres
    dims = 2 if case["two_d"] else 3
    c0 = math.sqrt(2 * case["gas"]["R"] * float(np.mean(case["T0"])))
    case["rho0"] = case["rho0"] * (1 + 0.05 * _smooth(rng, x, dims))
    case["T0"] = case["T0"] * (1 + 0.1 * _smooth(rng, x, dims))
    U = np.zeros((len(x), 3))
    for k in range(dims):
        U[:, k] = 0.1 * c0 * _smooth(rng, x, dims)
    case["U0"] = U
    nI = len(case["mesh"]["neighbour"])
    for p in case["mesh"]["patches"]:
        if p["type"] == "wall":
            sl = slice(p["startFace"], p["startFace"] + p["nFaces"])
            b = slice(sl.start - nI, sl.stop - nI)
            case["Tb"][b] *= 1 + 0.018 * _smooth(rng, xf[sl], dims)
    return case


def _flow(case, seed):
    """The case dict and time step of one flow case."""
    if case["mesh"] == "channel":
        c = C.channel2d(nx=case["n"], ny=case["ny"], Kn=case["kn"], nxi=case["nxi"])
        g = _geometry(c["mesh"])
        return _perturb(c, seed, (g["C"], g["Cf"])), C.stable_dt(c)
    key = (case["mesh"], case["n"], case["kind"] in ("value", "tangent", "adjoint"))
    gas, rho0 = C.gas_from_kn(case["kn"])
    c0 = math.sqrt(2 * gas["R"] * 273.0)
    c = C.make_case(_mesh(*key), gas, rho0, case["nxi"], 4.0 * c0, two_d=case["mesh"] != "hexes",
                    grid=case["grid"], C_gh=c0 if case["grid"] == "gh" else None)
    c["unstructured"] = case["mesh"] == "triangles"
    return _perturb(c, seed, _centres(*key)), C.case_dt(c)


def _batch_flows(case, seed):
    out = []
    for i, inst in enumerate(C.batch_instances(case["count"])):
        c = C.batch_case(inst)
        g = _geometry(c["mesh"])
        out.append((_perturb(c, seed * 1000 + i, (g["C"], g["Cf"])), C.stable_dt(c)))
    return out


def _patch(c, name):
    return [p["name"] for p in c["mesh"]["patches"]].index(name)


def _pinned(n):
    return {k: torch.empty((n, 3) if k in "Uq" else n, dtype=torch.float64, pin_memory=True).numpy() for k in FIELDS}


def prepare(case, seed):
    if case["kind"] == "batch":
        flows = _batch_flows(case, seed)
        b = solver.Batch([c for c, _ in flows], autotune=False, persistent=case["persistent"])
        for i, (_, dt) in enumerate(flows):
            b.set_dt(i, dt)
        return dict(case=case, batch=b)
    c, dt = _flow(case, seed)
    s = solver.FvDVM(c, precision=solver.FP32_FP64MOM if case["fp"] == 32 else solver.FP64)
    s.set_dt(dt)
    s.evolution(case.get("spinup", 0))
    state = dict(case=case, solver=s, dt=dt, out=_pinned(s.nCells))
    if case["kind"] in ("value", "tangent", "adjoint"):
        state["objective"] = dict(n_steps=case["steps"], avg_first=case["first"], q_patch=_patch(c, "movingWall"),
                                  stress_patch=_patch(c, "bottomWall"), checkpoint_every=case["every"])
        state["direction"] = np.random.default_rng(seed + 1).standard_normal(s.info()["n_wall_faces"])
    return state


# ------------------------------------------------------------------ one pass
def _fields(fp, out):
    """The cell fields as a post-processor keeps them: single precision for an FP32 run."""
    return {k: torch.from_numpy(out[k]).to(torch.float32) if fp == 32 else torch.from_numpy(out[k]) for k in FIELDS}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        b = state["batch"]
        b.step(case["steps"])
        b.synchronize()
        m = [b.macros(i) for i in range(case["count"])]
        return {k: torch.from_numpy(np.concatenate([x[k] for x in m])).to(torch.float32) for k in FIELDS}
    s, out = state["solver"], state["out"]
    if kind == "value":
        return dict(J=np.float64(s.objective_value(**state["objective"])))
    if kind == "tangent":
        J, dJ = s.objective_tangent(state["direction"], 1.0, **state["objective"])
        return dict(J=np.float64(J), dJ=np.float64(dJ))
    if kind == "adjoint":
        J, g, gs = s.objective_adjoint(**state["objective"])
        return dict(J=np.float64(J), dJdTw=torch.from_numpy(g.copy()), dJds=np.float64(gs))
    if kind == "loop":
        for _ in range(case["steps"]):
            s.getCoNum()
            s.set_dt(state["dt"])
            s.evolution(1)
        s.residual()
    else:
        s.evolution(case["steps"])
    s.macros_into(out["rho"], out["U"], out["T"], out["q"])
    return _fields(case["fp"], out)


# ------------------------------------------------------------------ work
def _size(case):
    """(cells, velocities, active faces, directions, fields) of a flow case."""
    if case["mesh"] == "triangles":
        n = case["n"]
        return 2 * n * n, case["nxi"] ** 2, 3 * n * n + 2 * n, 2, 2
    if case["mesh"] == "hexes":
        n = case["n"] ** 3
        return n, case["nxi"] ** 3, 3 * n + 3 * case["n"] ** 2, 3, 1
    nx, ny = case["n"], case.get("ny", case["n"])
    return nx * ny, case["nxi"] ** 2, 2 * nx * ny + nx + ny, 2, 2


def work(case):
    """Bytes: the distributions read and written once per step, the fields once per pass.  Operations per cell and
    velocity: one relaxation (about 20 + 10 per field) for the cell and for each face, gradient and reconstruction
    (4 D per face and field), flux (2 D + 2 per face side) and the moments of cells and faces."""
    if case["kind"] == "batch":
        by = fl = 0
        for i in C.batch_instances(case["count"]):
            w = work(dict(kind="steps", mesh="quads", n=i["N"], nxi=i["M"], fp=32, steps=case["steps"]))
            by, fl = by + w["bytes"], fl + w["flops"]
        return dict(bytes=by, flops=fl)
    nC, nV, nA, D, F = _size(case)
    e = case["fp"] // 8
    steps = case["steps"] * {"tangent": 2, "adjoint": 3}.get(case["kind"], 1)
    per_cell = 20 + 10 * F + 2 * (3 + 3 * D) * F
    per_face = (20 + 10 * F) + 8 * D * F + 2 * (2 * D + 2 * F) + 2 * (3 + 3 * D) * F
    return dict(bytes=steps * nV * nC * 2 * F * e + nC * 64, flops=steps * nV * (nC * per_cell + nA * per_face))


# ------------------------------------------------------------------ the step in 64 bits, from the equations alone
def _geometry(mesh):
    """Face centres and areas, cell centres and volumes of a polyhedral mesh (triangle fans and pyramids)."""
    pts, off, fv = mesh["points"], np.asarray(mesh["face_offsets"]), np.asarray(mesh["face_verts"])
    own, nei, nC = np.asarray(mesh["owner"]), np.asarray(mesh["neighbour"]), mesh["n_cells"]
    nF, nI = len(off) - 1, len(nei)
    Cf, Sf = np.zeros((nF, 3)), np.zeros((nF, 3))
    cnt = np.diff(off)
    for k in np.unique(cnt):
        f = np.nonzero(cnt == k)[0]
        P = pts[fv[off[f][:, None] + np.arange(k)]]
        if k == 3:
            Cf[f] = P.mean(1)
            Sf[f] = 0.5 * np.cross(P[:, 1] - P[:, 0], P[:, 2] - P[:, 0])
            continue
        m = P.mean(1)
        Q = np.roll(P, -1, axis=1)
        nrm = 0.5 * np.cross(Q - P, m[:, None] - P)
        mag = np.linalg.norm(nrm, axis=2)
        Sf[f] = nrm.sum(1)
        Cf[f] = ((P + Q + m[:, None]) / 3 * mag[..., None]).sum(1) / mag.sum(1)[:, None]
    est, num = np.zeros((nC, 3)), np.zeros(nC)
    for idx, sl in ((own, slice(0, nF)), (nei, slice(0, nI))):
        np.add.at(est, idx, Cf[sl])
        np.add.at(num, idx, 1.0)
    est /= num[:, None]
    V, M = np.zeros(nC), np.zeros((nC, 3))
    for idx, sl, sign in ((own, slice(0, nF), 1.0), (nei, slice(0, nI), -1.0)):
        h = sign * (Sf[sl] * (Cf[sl] - est[idx])).sum(1)
        np.add.at(V, idx, h)
        np.add.at(M, idx, h[:, None] * (0.75 * Cf[sl] + 0.25 * est[idx]))
    return dict(Cf=Cf, Sf=Sf, C=M / V[:, None], V=V / 3)


class _Flow64:
    """The DUGKS step on torch float64 tensors [entity, velocity]; walls (diffuse) and pressure patches."""

    def __init__(self, c, dt, dev):
        m, g, nI = c["mesh"], _geometry(c["mesh"]), len(c["mesh"]["neighbour"])
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
        ix = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.int64, device=dev)  # noqa: E731
        self.dev, self.dt, self.nC, self.nI = dev, dt, m["n_cells"], nI
        self.D = D = 2 if c["two_d"] else 3
        gas = c["gas"]
        self.R, self.om, self.Tref, self.mu, self.Pr, self.K = (gas[k] for k in ("R", "omega", "Tref", "muRef", "Pr", "KInner"))
        act = [p for p in m["patches"] if p["type"] != "empty"]
        bf = np.concatenate([np.arange(p["startFace"], p["startFace"] + p["nFaces"]) for p in act])
        self.kind = ix(np.concatenate([np.full(p["nFaces"], {"pressureIn": 1, "pressureOut": 2}.get(p.get("bc"), 0)) for p in act]))
        self.pB = t(np.concatenate([np.full(p["nFaces"], p.get("pressure", 0.0)) for p in act]))
        self.spans, at = {}, 0
        for p in act:
            self.spans[p["name"]] = slice(at, at + p["nFaces"])
            at += p["nFaces"]
        fs = np.concatenate([np.arange(nI), bf])
        self.own, self.nei = ix(np.asarray(m["owner"])[fs]), ix(m["neighbour"])
        o, n = np.asarray(m["owner"])[fs], np.asarray(m["neighbour"])
        S, Cf, Cc = g["Sf"][fs], g["Cf"][fs], g["C"]
        mag = np.linalg.norm(S, axis=1)
        nh = S / mag[:, None]
        d = np.empty((len(fs), 3))
        d[:nI] = Cc[n] - Cc[o[:nI]]
        d[nI:] = nh[nI:] * ((Cf[nI:] - Cc[o[nI:]]) * nh[nI:]).sum(1)[:, None]
        d2 = (d * d).sum(1)
        A = np.zeros((self.nC, 3, 3))
        w = d[:, :, None] * d[:, None, :] / d2[:, None, None]
        np.add.at(A, o, w)
        np.add.at(A, n, w[:nI])
        A = np.linalg.inv(A[:, :D, :D])
        L = d[:, :D] / d2[:, None]
        self.Lo, self.Ln = t(np.einsum("fij,fj->fi", A[o], L)), t(np.einsum("fij,fj->fi", A[n], L[:nI]))
        self.inv_dc = t(np.sqrt(d2[nI:]))[:, None]
        self.nb = t(nh[nI:])
        self.S, self.magB, self.V = t(S), t(mag[nI:]), t(g["V"])
        self.dO, self.dN = t(Cf - Cc[o]), t(Cf[:nI] - Cc[n])
        x, w1 = np.asarray(c["xis"]), np.asarray(c["weights"])
        grids = np.meshgrid(*([x] * D), indexing="ij")[::-1]
        ws = np.meshgrid(*([w1] * D), indexing="ij")
        self.xi = [t(a.ravel()) for a in grids]
        self.w = t(np.prod(ws, axis=0).ravel())
        bi = bf - nI
        self.Tb, self.Ub, self.rhob = t(c["Tb"][bi]), t(c["Ub"][bi]), t(np.zeros(len(bf)))
        self.rho, self.U, self.T = t(c["rho0"]), t(c["U0"])[:, :D], t(c["T0"])
        self.q = torch.zeros_like(self.U)
        self.scale = torch.ones((), dtype=torch.float64, device=dev)

    def start(self):
        self.tau = self._tau(self.rho, self.T)
        self.g, self.h = self._shakhov(self.rho, self.U, self.T, self.q)
        self.Gg = torch.zeros((len(self.Tb), len(self.w)), dtype=torch.float64, device=self.dev)
        self.Gh = torch.zeros_like(self.Gg)
        if bool((self.kind > 0).any()):
            self._pressure()

    def _tau(self, rho, T):
        return self.mu * self.scale * (T / self.Tref) ** self.om / (rho * self.R * T)

    def _c(self, U):
        return [x[None, :] - U[:, k, None] for k, x in enumerate(self.xi)]

    def _shakhov(self, rho, U, T, q):
        D, K = self.D, self.K
        RT = (self.R * T)[:, None]
        c2, cq = 0.0, 0.0
        for k, x in enumerate(self.xi):
            c = x[None, :] - U[:, k, None]
            c2 = c2 + c * c
            cq = cq + c * q[:, k, None]
        c2 = c2 / RT
        s = (1 - self.Pr) * cq / (5 * rho[:, None] * RT * RT)
        e = rho[:, None] * (2 * math.pi * RT) ** (-D / 2) * torch.exp(-0.5 * c2)
        g = e * (1 + s * (c2 - D - 2))
        if K + 3 - D == 0:
            return g, None
        return g, e * RT * ((K + 3 - D) + s * ((c2 - D) * (K + 3 - D) - 2 * K))

    def _maxwell(self, U, T):
        RT = (self.R * T)[:, None]
        c2 = 0.0
        for k, x in enumerate(self.xi):
            c2 = c2 + (x[None, :] - U[:, k, None]) ** 2
        return (2 * math.pi * RT) ** (-self.D / 2) * torch.exp(-c2 / (2 * RT))

    def _macros(self, g, h, facA):
        w = self.w
        rho = g @ w
        U = torch.stack([g @ (w * x) for x in self.xi], 1) / rho[:, None]
        x2 = sum(x * x for x in self.xi)
        E = 0.5 * (g @ (w * x2)) + (0.5 * (h @ w) if h is not None else 0.0)
        T = (E - 0.5 * rho * (U * U).sum(1)) / ((self.K + 3) / 2.0 * self.R * rho)
        tau = self._tau(rho, T)
        c = self._c(U)
        s = sum(a * a for a in c) * g
        if h is not None:
            s = s + h
        s = 0.5 * w * s
        q = torch.stack([(a * s).sum(1) for a in c], 1) * (2 * tau / (2 * tau + facA))[:, None]
        return rho, U, T, q, tau

    def _gradient(self, f, G):
        df = f[self.nei] - f[self.own[: self.nI]]
        db = G * self.inv_dc
        out = []
        for k in range(self.D):
            gk = torch.zeros_like(f).index_add(0, self.own[: self.nI], self.Lo[: self.nI, k, None] * df)
            gk = gk.index_add(0, self.nei, self.Ln[:, k, None] * df)
            out.append(gk.index_add(0, self.own[self.nI:], self.Lo[self.nI:, k, None] * db))
        Gn = sum(out[k][self.own[self.nI:]] * self.nb[:, k, None] for k in range(self.D))
        return out, Gn

    def _recon(self, f, grad, up):
        def side(cell, d):
            v = f[cell]
            for k in range(self.D):
                v = v + grad[k][cell] * (d[:, k, None] - 0.5 * self.dt * self.xi[k][None, :])
            return v

        vo = side(self.own, self.dO)
        vn = side(self.nei, self.dN)
        inner = torch.where(up[: self.nI] > 0, vo[: self.nI], torch.where(up[: self.nI] < 0, vn, 0.5 * (vo[: self.nI] + vn)))
        return torch.cat([inner, vo[self.nI:]])

    def _pressure(self):
        i, o = self.kind > 0, self.own[self.nI:]
        n, Ui, Ti, ri = self.nb, self.U[o], self.T[o], self.rho[o]
        a = torch.sqrt(self.R * Ti * (self.K + 5) / (self.K + 3))
        Un = (Ui * n[:, : self.D]).sum(1)
        dp = self.pB - ri * self.R * Ti
        inlet = self.kind == 1
        rb = torch.where(inlet, self.pB / (self.R * self.Tb), ri + dp / (a * a))
        self.rhob = torch.where(i, rb, self.rhob)
        self.Tb = torch.where(i & ~inlet, self.pB / (self.R * ri), self.Tb)

    def step(self, weights=None):
        dt, nI, own, nei = self.dt, self.nI, self.own, self.nei
        rf = (1.5 * dt / (2 * self.tau + dt))[:, None]
        ge, he = self._shakhov(self.rho, self.U, self.T, self.q)
        gB = (1 - rf) * self.g + rf * ge
        hB = None if he is None else (1 - rf) * self.h + rf * he
        del ge, he
        xs = sum(self.S[:, k, None] * x[None, :] for k, x in enumerate(self.xi))
        grad, self.Gg = self._gradient(gB, self.Gg)
        gS = self._recon(gB, grad, xs)
        hS = None
        if hB is not None:
            grad, self.Gh = self._gradient(hB, self.Gh)
            hS = self._recon(hB, grad, xs)
        del grad
        # boundary faces: incoming velocities
        xb, gb = xs[nI:], gS[nI:]
        outgoing = xb > 0
        Mw = self._maxwell(self.Ub[:, : self.D], self.Tb)
        inc = torch.abs((torch.where(xb < 0, -xb * Mw, torch.zeros_like(Mw))) @ self.w)
        rw = torch.where(outgoing, xb * gb, torch.zeros_like(gb)) @ self.w / inc
        gin = rw[:, None] * Mw
        open_ = self.kind > 0
        if bool(open_.any()):
            far = self.rhob[:, None] * self._maxwell(self.U[own[nI:]], self.Tb)
            gin = torch.where(open_[:, None], far, gin)
        gS = torch.cat([gS[:nI], torch.where(outgoing, gb, gin)])
        if hS is not None:
            hin = gin * (self.R * self.Tb * (self.K + 3 - self.D))[:, None]
            hS = torch.cat([hS[:nI], torch.where(outgoing, hS[nI:], hin)])
        rho, U, T, q, tau = self._macros(gS, hS, 0.5 * dt * self.Pr)
        J = 0.0
        if weights is not None:  # wall heat flux on the lid, shear on the bottom
            wq, ws = weights
            tw = tau[nI:]
            x2 = sum((x[None, :] - self.Ub[:, k, None]) ** 2 for k, x in enumerate(self.xi))
            e = 0.5 * self.w * (x2 * gS[nI:] + (hS[nI:] if hS is not None else 0.0))
            for k, x in enumerate(self.xi):
                qk = 2 * tw / (2 * tw + 0.5 * dt * self.Pr) * (e * (x[None, :] - self.Ub[:, k, None])).sum(1)
                J = J + (wq[:, k] * qk).sum()
            J = J + (ws * 2 * tw / (2 * tw + 0.5 * dt) * (gS[nI:] @ (self.w * self.xi[0] * self.xi[1]))).sum()
        b = (0.5 * dt / (2 * tau + 0.5 * dt))[:, None]
        ge, he = self._shakhov(rho, U, T, q)
        keep = torch.cat([torch.zeros((nI, 1), dtype=torch.bool, device=self.dev).expand(nI, len(self.w)), ~outgoing])
        gS = torch.where(keep, gS, (1 - b) * gS + b * ge)
        k = (dt / self.V)[:, None]

        def update(f, fB, fS):
            flux = xs * fS
            s = torch.zeros_like(f).index_add(0, own, -flux).index_add(0, nei, flux[:nI])
            return -f / 3 + 4 * fB / 3 + k * s

        if hS is not None:
            hS = torch.where(keep, hS, (1 - b) * hS + b * he)
            self.h = update(self.h, hB, hS)
        del ge, he
        self.g = update(self.g, gB, gS)
        self.rho, self.U, self.T, self.q, self.tau = self._macros(self.g, self.h, dt * self.Pr)
        if bool(open_.any()):
            self._pressure()
        return J

    def fields(self):
        pad = lambda a: torch.nn.functional.pad(a, (0, 3 - self.D))  # noqa: E731
        return dict(rho=self.rho, U=pad(self.U), T=self.T, q=pad(self.q))


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "batch":
        with torch.no_grad():
            parts = []
            for c, dt in _batch_flows(case, seed):
                f = _Flow64(c, dt, dev)
                f.start()
                for _ in range(case["steps"]):
                    f.step()
                parts.append(f.fields())
            return {k: torch.cat([p[k] for p in parts]).cpu() for k in FIELDS}
    c, dt = _flow(case, seed)
    f = _Flow64(c, dt, dev)
    if case["kind"] in ("steps", "loop"):
        steps = case.get("spinup", 0) + case["steps"]
        if f.nC * len(f.w) * max(steps, 6) > 2.5e9:
            return None  # the largest flows: over 20 seconds, or hundreds of GB, in 64 bits
        with torch.no_grad():
            f.start()
            for _ in range(steps):
                f.step()
            return {k: v.cpu() for k, v in f.fields().items()}
    grad = case["kind"] != "value"
    f.Tb.requires_grad_(grad)
    f.scale.requires_grad_(grad)
    nB = len(f.Tb)
    wq, ws = torch.zeros((nB, 3), dtype=torch.float64, device=dev), torch.zeros(nB, dtype=torch.float64, device=dev)
    lid, low = f.spans["movingWall"], f.spans["bottomWall"]
    wq[lid] = f.S[f.nI:][lid]
    ws[low] = f.magB[low]
    J = 0.0
    with torch.set_grad_enabled(grad):
        f.start()
        for n in range(case["steps"]):
            J = J + f.step((wq, ws) if n >= case["first"] else None)
        J = J / (case["steps"] - case["first"])
    if not grad:
        return dict(J=np.float64(J))
    gT, gs = torch.autograd.grad(J, [f.Tb, f.scale])
    if case["kind"] == "adjoint":
        return dict(J=np.float64(J.item()), dJdTw=gT.cpu(), dJds=np.float64(gs.item()))
    d = torch.as_tensor(np.random.default_rng(seed + 1).standard_normal(nB), device=dev)
    return dict(J=np.float64(J.item()), dJ=np.float64(((gT * d).sum() + gs).item()))
