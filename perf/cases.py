"""The work a user of this package has it do, as cases that can be timed and checked.

A case is a mesh (cantilever bar, voxel vertebral body of TET4 or HEX8
elements, motion segment), a material and one call of the public API:

``forces``   ``material.compute_nodal_forces(mesh)``: the residual pass of
             every Newton iteration and of explicit dynamics
``stress``   ``material.compute_stress`` and the nodal von Mises stress: what
             a program exports after a solve
``tangent``  ``fem_tangent_matvec``: one product with the consistent tangent
             (Newmark steps, arc-length predictors, a caller's own Krylov loop)
``network``  ``fem_mpnn_forward``: the learned preconditioner's forward pass
``solve``    ``StaticSolver.solve()`` with the library's defaults, one load step
``path``     the benchmark's loop: load steps from rest with the tuned options
             (4-voxel lattice, BF16 inverse, load-step extrapolation)
``batch``    ``solve_batch`` over bodies of uneven size

``exact`` gives the same results in plain 64-bit torch (solves only where a
dense factorisation is small).
"""
from __future__ import annotations

import ctypes as C
import functools
import math
import random

import numpy as np
import torch

from simul_b200 import _lib, batch, learned, meshgen
from simul_b200 import fem as B

NU, SIGMA_Y = 0.3, 100.0
MR = (0.18, 0.045, 0.5)               # C10, C01, D1 of the Mooney-Rivlin bar
DISC = (0.18, 0.045, 2.0 / 4.5)       # the segment's disc matrix
DENSE_MAX = 4500                      # unknowns up to which exact() solves
TOL = 1e-10                           # of the solves: displacements settled well below what a result file keeps


def listed():
    return [
        # the README's bar (1,920 tets): launches and synchronisation are what it costs
        {"name": "bar_forces", "op": "forces", "mesh": "bar", "n": 4, "material": "nh"},
        {"name": "bar_solve", "op": "solve", "mesh": "bar", "n": 4, "material": "nh"},
        # the benchmark's body: 64 voxels per axis, 566,000 tets, J2 bone
        {"name": "body64_forces", "op": "forces", "mesh": "tet4", "n": 64, "material": "j2"},
        {"name": "body64_stress", "op": "stress", "mesh": "tet4", "n": 64, "material": "j2"},
        # an odd size above the benchmark's (the 1M-tet point)
        {"name": "body78_tangent", "op": "tangent", "mesh": "tet4", "n": 78, "material": "j2"},
        # a first solve as the README writes it, nothing tuned
        {"name": "body48_solve", "op": "solve", "mesh": "tet4", "n": 48, "material": "j2"},
        # the headline: 20 load steps from rest
        {"name": "body64_path", "op": "path", "mesh": "tet4", "n": 64, "material": "j2", "steps": 20},
        # bone, disc and screw on one mesh: mixed material table, forces as loads
        {"name": "segment16_solve", "op": "solve", "mesh": "segment", "n": 16, "material": "mixed"},
        {"name": "hex64_forces", "op": "forces", "mesh": "hex8", "n": 64, "material": "j2"},
        {"name": "hex48_path", "op": "path", "mesh": "hex8", "n": 48, "material": "j2", "steps": 10},
        {"name": "body48_network", "op": "network", "mesh": "tet4", "n": 48, "material": "j2"},
        # the batch workload's sizes, fewer of them
        {"name": "batch8", "op": "batch", "mesh": "tet4", "n": 32, "n_max": 56, "count": 8, "material": "j2",
         "steps": 5},
    ]


def draw(rng: random.Random):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["forces", "forces", "stress", "tangent", "tangent", "network", "solve", "solve", "path", "path",
                     "batch"])
    if op == "batch":
        n = log_int(16, 40)
        return {"op": op, "mesh": "tet4", "n": n, "n_max": n + rng.randint(2, 16), "count": rng.randint(2, 8),
                "material": "j2", "steps": rng.randint(2, 5)}
    if op == "path":
        mesh = rng.choice(["tet4", "tet4", "hex8"])
        return {"op": op, "mesh": mesh, "n": log_int(14, 60 if mesh == "tet4" else 48), "material": "j2",
                "steps": rng.randint(3, 20)}
    if op == "network":
        return {"op": op, "mesh": "tet4", "n": log_int(12, 56), "material": "j2"}
    if op == "solve":
        mesh = rng.choice(["bar", "tet4", "hex8"])
        if mesh == "bar":
            return {"op": op, "mesh": mesh, "n": log_int(2, 12), "material": rng.choice(["nh", "le"])}
        return {"op": op, "mesh": mesh, "n": log_int(12, 56), "material": rng.choice(["j2", "le"])}
    mesh = rng.choice(["bar", "tet4", "tet4", "hex8"])
    if mesh == "bar":
        return {"op": op, "mesh": mesh, "n": log_int(2, 24), "material": rng.choice(["nh", "mr", "le"])}
    return {"op": op, "mesh": mesh, "n": log_int(12, 90 if mesh == "tet4" else 72),
            "material": rng.choice(["j2", "j2", "nh", "le"])}


# ───────────────────────── inputs ─────────────────────────

@functools.lru_cache(maxsize=8)
def _geometry(kind, n, seed):
    """Mesh, moduli, constraints and full-load values of one body."""
    if kind == "bar":
        v = meshgen.cantilever_bar(5 * n, n, n)
        v.E = np.full(v.n_elements, 17e3)
    elif kind == "segment":
        v = meshgen.motion_segment(n=n, seed=seed)
    else:
        v = meshgen.vertebral_body(n=n, seed=seed, element=kind)
    # the library stores moduli as a 32-bit scale of the first one
    v.E = v.E[0] * (v.E / v.E[0]).astype(np.float32).astype(np.float64)
    return v


def _body(case, seed):
    return _geometry(case["mesh"], case["n"], seed if case["mesh"] != "bar" else 0)


def _specs(case, seed):
    """(grid size, seed) of the instances of a batch: sizes spread over [n, n_max]."""
    last = max(case["count"] - 1, 1)
    return [(case["n"] + (case["n_max"] - case["n"]) * i // last, seed + i) for i in range(case["count"])]


def _material(case, v):
    kind = case["material"]
    E = float(v.E[0]) if case["mesh"] == "bar" else v.E
    if kind == "nh":
        return B.NeoHookean(E, NU)
    if kind == "le":
        return B.LinearElastic(E, NU)
    if kind == "mr":
        return B.MooneyRivlin(*MR)
    j2 = B.J2Plasticity(v.E, NU, SIGMA_Y, hardening_modulus=0.02 * v.E)
    if kind == "mixed":
        return {0: j2, 1: B.MooneyRivlin(*DISC), 2: B.LinearElastic(110e3, NU)}
    return j2


def _displacements(v, case, seed):
    """Two displacement fields: a loaded state whose plastic history is kept,
    and the state the call is made at.  The body is compressed past yield."""
    g = np.random.default_rng(seed)
    h = (np.ptp(v.X[:, 0]) * np.ptp(v.X[:, 1]) * np.ptp(v.X[:, 2]) / v.n_nodes) ** (1.0 / 3.0)
    out = []
    for strain in (0.006, 0.009):
        u = 1e-3 * h * g.standard_normal(v.X.shape)
        k = g.uniform(0.5, 2.0, 3) * np.pi / np.ptp(v.X, axis=0)
        u += 2e-3 * np.ptp(v.X[:, 2]) * np.sin(v.X @ k)[:, None] * g.uniform(-0.3, 0.3, 3)
        u[:, 2] -= strain * v.X[:, 2]
        out.append(u)
    return out


def _load(case, v, seed):
    """Full prescribed values and forces of the solve."""
    s = 1.0 + 0.1 * np.random.default_rng(seed).uniform(-1.0, 1.0)
    if case["op"] == "solve":  # one step into the plastic range
        s *= 0.4
    f = v.f_ext * (0.25 * s)
    if case["mesh"] == "segment":
        f = meshgen.top_moment_forces(v.X, np.isclose(v.X[:, 2], v.X[:, 2].max()), "flexion", 125.0 * s)
    return v.fixed_vals * s, f


def _mesh(case, v):
    mesh = B.FEMesh(v.n_nodes, v.n_elements, B.ElementType.HEX8 if case["mesh"] == "hex8" else B.ElementType.TET4)
    mesh.initialize_from_numpy(v.X, v.conn, material_ids=v.info.get("material_ids"))
    return mesh


def _cuda(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a)).to("cuda", dtype)


def _weights(seed):
    return learned.init_weights(seed=seed, out_scale=0.2)


def _vector(v, seed):
    r = np.random.default_rng(seed + 1).standard_normal(v.X.shape)
    r[v.fixed_mask] = 0.0
    return r.astype(np.float32)


def prepare(case, seed):
    op = case["op"]
    if op == "batch":
        insts = []
        for n, s in _specs(case, seed):
            v = _geometry("tet4", n, s)
            inst = batch.BatchInstance(v.X, v.conn, _material(case, v), v.fixed_mask, v.fixed_vals, coarse_cell=4,
                                       coarse_bf16=True, coarse_reuse=0)
            inst.mesh.set_extrapolation(True)
            insts.append(inst)
        return {"op": op, "insts": insts, "steps": case["steps"]}
    v = _body(case, seed)
    mesh, mat = _mesh(case, v), _material(case, v)
    st = {"op": op, "mesh": mesh, "mat": mat}
    if op in ("solve", "path"):
        vals, f = _load(case, v, seed)
        fixed = np.where(v.fixed_mask.reshape(-1))[0]
        mesh.set_fixed_dofs(fixed)
        st.update(vals=_cuda(vals), f=_cuda(f), steps=case.get("steps", 1), j2=case["material"] == "j2")
        kw = {"materials": mat} if isinstance(mat, dict) else {"material": mat}
        st["solver"] = B.StaticSolver(mesh, tol=TOL, **kw)
        if op == "path":
            mesh.set_coarse_options(cell=4, bf16=True, reuse=0, inverse="tf32", max_nodes=6144)
            mesh.set_extrapolation(True)
        return st
    mesh.set_fixed_dofs(np.where(v.fixed_mask.reshape(-1))[0])
    u0, u1 = _displacements(v, case, seed)
    if case["material"] == "j2":  # a committed plastic state
        mesh.u.copy_(_cuda(u0))
        mat.compute_nodal_forces(mesh)
        B._check(_lib.load().fem_commit_history(mesh.ctx), mesh.ctx, "fem_commit_history")
    mesh.u.copy_(_cuda(u1))
    if op in ("tangent", "network"):
        mat.compute_nodal_forces(mesh)
        st["x"] = _cuda(_vector(v, seed), torch.float32)
        st["y"] = torch.empty_like(st["x"])
        if op == "network":
            learned.set_weights(mesh, _weights(seed))
    return st


# ───────────────────────── one pass ─────────────────────────

def run(state):
    op = state["op"]
    if op == "batch":
        for inst in state["insts"]:
            inst.reset()
        batch.solve_batch(state["insts"], load_steps=state["steps"], tol=TOL)
        return {"u": [inst.mesh.u for inst in state["insts"]]}
    mesh, mat = state["mesh"], state["mat"]
    if op == "forces":
        mat.compute_nodal_forces(mesh)
        return {"f": mesh.f}
    if op == "stress":
        mat.compute_stress(mesh)
        mesh.compute_mises_stress()
        return {"F": mesh.F, "stress": mesh.stress, "mises": mesh.mises}
    if op in ("tangent", "network"):
        lib = _lib.load()
        fn = lib.fem_tangent_matvec if op == "tangent" else lib.fem_mpnn_forward
        B._check(fn(mesh.ctx, B._ptr(state["x"]), B._ptr(state["y"])), mesh.ctx, op)
        return {"y": state["y"]}
    # a load path from rest
    mesh.u.zero_()
    if state["j2"]:
        mat.reset_state()
    for k in range(1, state["steps"] + 1):
        load = k / 20 if state["op"] == "path" else 1.0
        torch.mul(state["vals"], load, out=mesh.fixed_value)
        torch.mul(state["f"], load, out=mesh.f_ext)
        mesh._bc_dirty = True
        state["solver"].solve(verbose=False)
    return {"u": mesh.u}


def work(case):
    """Bytes: mesh, moduli, fields and history in, results out (of each load
    step); flops: of the element passes (the solves' iterations not counted)."""
    total = {"bytes": 0.0, "flops": 0.0}
    for n, s in _specs(case, 0) if case["op"] == "batch" else [(case["n"], 0)]:
        v = _geometry(case["mesh"], n, 0)
        ne, nn = v.n_elements, v.n_nodes
        npe, nq = v.conn.shape[1], v.n_elements * (8 if case["mesh"] == "hex8" else 1)
        small = case["material"] in ("j2", "le")
        state = {"j2": 32, "nh": 40, "mr": 36, "le": 0, "mixed": 36}[case["material"]]  # tangent words of a point
        hist = 56 if case["material"] == "j2" else 0
        b = ne * (4 * npe + 4)
        if case["op"] == "forces":
            b += nn * (24 + 24 + 24) + nq * (2 * hist + state)
        elif case["op"] == "stress":
            b += nn * (24 + 24 + 8) + nq * (hist + 144)
        elif case["op"] == "tangent":
            b += nn * (12 + 12 + 12) + nq * state
        elif case["op"] == "network":
            b += nn * (12 + 12 + 12) + nq * state + 4 * _lib.MPNN_PARAMS
        else:
            b += case.get("steps", 1) * (nn * (24 + 24 + 24) + nq * (2 * hist + state))
        f = nq * (30.0 * npe + (150.0 if small else 300.0)) * case.get("steps", 1)
        if case["op"] == "network":
            f = nn * 2.0 * (16 * 64 + 4 * 128 * 64 + 64 * 3)
        total["bytes"] += b
        total["flops"] += f
    return total


# ───────────────────────── the same in 64 bits ─────────────────────────

class _Plain:
    """Element forces and tangents in plain 64-bit torch."""

    def __init__(self, v, case):
        self.X, self.conn = _cuda(v.X), _cuda(v.conn, torch.int64)
        self.E, self.kind = _cuda(v.E)[:, None], case["material"]
        Xe = self.X[self.conn]
        if self.conn.shape[1] == 4:
            d = torch.tensor([[[-1.0, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]]], dtype=torch.float64, device="cuda")
            weight = 1.0 / 6.0
        else:
            s = torch.tensor(meshgen.HEX8_CORNERS, dtype=torch.float64, device="cuda")
            f = 1.0 + s[None] * (s[:, None] * 0.5773502691896257)         # point, vertex, axis
            d = 0.125 * torch.stack([s[:, 0] * f[..., 1] * f[..., 2], s[:, 1] * f[..., 0] * f[..., 2],
                                     s[:, 2] * f[..., 0] * f[..., 1]], dim=-1)
            weight = 1.0
        J = torch.einsum("eai,qaj->eqij", Xe, d)
        self.dN = torch.einsum("qaj,eqjk->eqak", d, torch.linalg.inv(J))
        self.w = weight * torch.linalg.det(J).abs()
        self.hist = None
        if self.kind == "j2":
            self.hist = (torch.zeros(J.shape, dtype=torch.float64, device="cuda"), torch.zeros_like(self.w))

    def stress(self, H, E, hist, cauchy=False):
        """The stress contracted with dN/dX (first Piola-Kirchhoff for the
        large-strain models), or the Cauchy stress; J2 also its new history."""
        mu, lam = E / (2 * (1 + NU)), E * NU / ((1 + NU) * (1 - 2 * NU))
        eye = torch.eye(3, dtype=torch.float64, device=H.device)
        mu, lam = mu[..., None, None], lam[..., None, None]
        if self.kind in ("nh", "mr"):
            F = eye + H
            J = torch.linalg.det(F)[..., None, None]
            Ft = torch.linalg.inv(F).transpose(-1, -2)
            if self.kind == "nh":
                P = mu * (F - Ft) + lam * torch.log(J) * Ft
            else:
                Bm = F @ F.transpose(-1, -2)
                tr = torch.einsum("...ii->...", Bm)[..., None, None]
                P = 2 * (MR[0] + MR[1] * tr) * F - 2 * MR[1] * Bm @ F + 2 / MR[2] * J * J * (J - 1) * Ft
            return (P @ F.transpose(-1, -2) / J if cauchy else P), hist
        e = 0.5 * (H + H.transpose(-1, -2))
        if self.kind == "j2":
            ep, epe = hist
            e = e - ep
        tr = torch.einsum("...ii->...", e)[..., None, None] * eye
        s = lam * tr + 2 * mu * e
        if self.kind != "j2":
            return s, hist
        dev = 2 * mu * (e - tr / 3)
        norm = torch.sqrt((dev * dev).sum((-1, -2)).clamp_min(1e-30))
        f = math.sqrt(1.5) * norm - (SIGMA_Y + 0.02 * E * epe)
        dg = torch.clamp(f, min=0.0) / (3 * mu[..., 0, 0] + 0.02 * E)
        flow = math.sqrt(1.5) * dg[..., None, None] * dev / norm[..., None, None]
        return s - 2 * mu * flow, (ep + flow, epe + dg)

    def grad(self, u):
        return torch.einsum("eai,eqak->eqik", u[self.conn], self.dN)

    def _element(self, ue, dN, w, E, hist):
        S, _ = self.stress(torch.einsum("ai,qak->qik", ue, dN), E, hist)
        return -torch.einsum("q,qij,qaj->ai", w, S, dN)

    def forces(self, u):
        S, new = self.stress(self.grad(u), self.E, self.hist)
        fe = -torch.einsum("eq,eqij,eqaj->eai", self.w, S, self.dN)
        out = torch.zeros_like(u)
        out.index_add_(0, self.conn.reshape(-1), fe.reshape(-1, 3))
        return out, new

    def stiffness(self, u, size=65536):
        """Element stiffness matrices (elements, vertices, 3, vertices, 3), a block of elements at a time."""
        fn = torch.func.vmap(torch.func.jacfwd(self._element), in_dims=(0, 0, 0, 0, 0 if self.hist else None))
        for e in range(0, self.conn.shape[0], size):
            h = tuple(t[e:e + size] for t in self.hist) if self.hist else None
            s = slice(e, e + size)
            yield s, -fn(u[self.conn[s]], self.dN[s], self.w[s], self.E[s], h)

    def newton(self, u, fixed, vals, f_ext):
        free = torch.nonzero(~fixed.reshape(-1)).reshape(-1)
        n = u.numel()
        dof = (3 * self.conn[:, :, None] + torch.arange(3, device="cuda")).reshape(self.conn.shape[0], -1)
        first = None
        for it in range(30):
            R = (f_ext + self.forces(u)[0]).reshape(-1)
            du = torch.zeros(n, dtype=torch.float64, device="cuda")
            du[fixed.reshape(-1)] = (vals - u)[fixed]
            norm = float(R[free].norm())
            if it and norm <= 1e-13 * max(first, 1e-300):
                break
            K = torch.zeros(n * n, dtype=torch.float64, device="cuda")
            for s, k in self.stiffness(u):
                k = k.reshape(k.shape[0], -1)
                K.index_add_(0, (dof[s][:, :, None] * n + dof[s][:, None, :]).reshape(-1), k.reshape(-1))
            K = K.reshape(n, n)
            rhs = R - K @ du
            first = max(first or 0.0, float(rhs[free].norm()))
            du[free] = torch.linalg.solve(K[free][:, free], rhs[free])
            u = u + du.reshape(u.shape)
        return u


def _plain_path(case, v, vals, f, steps):
    p = _Plain(v, case)
    u, fixed = torch.zeros_like(p.X), _cuda(v.fixed_mask, torch.bool)
    vals, f = _cuda(vals), _cuda(f)
    for load in steps:
        u = p.newton(u, fixed, vals * load, f * load)
        if p.hist:
            p.hist = p.forces(u)[1]
    return u


def _plain_network(p, v, case, u, r, w):
    nn = v.n_nodes
    diag = torch.zeros(nn, 3, dtype=torch.float64, device="cuda")
    for s, k in p.stiffness(u):
        d = torch.diagonal(torch.diagonal(k, dim1=1, dim2=3), dim1=1, dim2=2)
        diag.index_add_(0, p.conn[s].reshape(-1), d.reshape(-1, 3))
    fixed = _cuda(v.fixed_mask, torch.bool)
    dinv = torch.where(fixed, 0.0, 1.0 / diag)
    pairs = torch.cat([p.conn[:, [a, b]] for a in range(4) for b in range(4) if a != b])
    pairs = torch.unique(pairs[:, 0] * nn + pairs[:, 1])
    row, col = pairs // nn, pairs % nn
    deg = torch.bincount(row, minlength=nn).clamp_min(1)[:, None]
    ones = torch.ones(p.conn.numel(), dtype=torch.float64, device="cuda")
    mod = (p.E * (1 - NU) / ((1 + NU) * (1 - 2 * NU))).expand(-1, 4).reshape(-1)
    total = torch.zeros(2, nn, dtype=torch.float64, device="cuda")
    total[0].index_add_(0, p.conn.reshape(-1), mod)
    total[1].index_add_(0, p.conn.reshape(-1), ones)
    c = torch.log(total[0] / total[1])
    d = dinv.sqrt()
    x = d * r
    s = torch.sqrt((x * x).sum() / nn)
    feat = torch.zeros(nn, 16, dtype=torch.float64, device="cuda")
    feat[:, :3], feat[:, 3:6], feat[:, 6] = x / s, fixed.double(), c - c.mean()
    w, at = _cuda(w), 0

    def take(*shape):
        nonlocal at
        at += math.prod(shape)
        return w[at - math.prod(shape):at].reshape(shape)

    h = torch.relu(feat @ take(64, 16).T + take(64))
    for _ in range(4):
        m = torch.zeros_like(h).index_add_(0, row, h[col]) / deg
        h = h + torch.relu(torch.cat([h, m], 1) @ take(64, 128).T + take(64))
    return dinv * r + s * d * (h @ take(3, 64).T + take(3))


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        return None
    v = _body(case, seed)
    if op in ("solve", "path"):
        if case["material"] == "mixed" or 3 * v.n_nodes > DENSE_MAX:
            return None
        vals, f = _load(case, v, seed)
        steps = [k / 20 if op == "path" else 1.0 for k in range(1, case.get("steps", 1) + 1)]
        return {"u": _plain_path(case, v, vals, f, steps)}
    p = _Plain(v, case)
    u0, u1 = (_cuda(u) for u in _displacements(v, case, seed))
    if p.hist:
        p.hist = p.forces(u0)[1]
    if op == "forces":
        return {"f": p.forces(u1)[0]}
    if op == "stress":
        H = p.grad(u1)
        s = p.stress(H, p.E, p.hist, cauchy=True)[0]
        m = s.mean(1)
        m = m - torch.einsum("eii->e", m)[:, None, None] / 3 * torch.eye(3, dtype=torch.float64, device="cuda")
        vm = torch.sqrt(1.5 * (m * m).sum((1, 2)))
        mises = torch.zeros(v.n_nodes, dtype=torch.float64, device="cuda")
        mises.index_add_(0, p.conn.reshape(-1), vm[:, None].expand(p.conn.shape).reshape(-1))
        return {"F": (torch.eye(3, dtype=torch.float64, device="cuda") + H).reshape(-1, 3, 3),
                "stress": s.reshape(-1, 3, 3), "mises": mises}
    x = _cuda(_vector(v, seed))
    if op == "network":
        return {"y": _plain_network(p, v, case, u1, x, _weights(seed))}
    fixed = _cuda(v.fixed_mask, torch.bool)
    y = -torch.func.jvp(lambda u: p.forces(u)[0], (u1,), (x,))[1]
    return {"y": torch.where(fixed, 0.0, y)}
