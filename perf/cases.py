"""The work that users of the framework have it do, as timed cases.

Every case goes through the public Python binding of the C ABI
(``flexmesh_b200.Context``) on the unit-cube workloads of
``flexmesh_b200/configs.py`` (or generic inputs where the entry point takes
any), from calls that finish in microseconds to one load step of the
benchmark's 64^3 block.  A case is a dict of plain values; ``prepare`` makes
what a program holds before the call (context with mesh, material, Dirichlet
data; device tensors), ``run`` makes the call, ``work`` counts the bytes and
operations the call cannot do without, and ``exact`` gives the same outputs
from plain FP64 torch.

Kinds
  assemble   tangent + internal force into the CSR (FP64 or FP32 tangent)
  residual   internal force only (what each line-search trial needs)
  elements   batched 12x12 tangents and forces of independent tets
  ilu_apply  ILU(0) factorization and one preconditioner apply, FP64
  pcg        ILU(0) factorization and PCG to 1e-12, FP64
  csr_pcg    the host-array PCG-ILU(0) on a generic CSR matrix
  newton     one load step, FP64 (parity settings) or mixed (bench settings)
  adjoint    material gradients of a loss on u (the backward direction)
  states     SL(3) element state update and Mandel stress
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "atlas-flexmesh_b200"))

import flexmesh_b200 as F  # noqa: E402
from flexmesh_b200 import configs  # noqa: E402

PREC = {"fp64": F.FM_FP64, "mixed": F.FM_MIXED}
# the benchmark's Newton settings; the residual is brought two decades lower
# (as the material-gradient workload's forward solves have it), so that u is
# determined to well below 1e-9 whatever the inner solves' rounding
MIXED = dict(newton_rtol=1e-12, inner_tol=0.8, predictor_tol=1e-6, max_newton=400,
             max_pcg=20000, line_search=10, ls_c=1e-4, initial_guess=1, ilu_every=3)
FP64 = dict(newton_rtol=1e-12, inner_tol=1e-12, max_newton=400, max_pcg=20000, line_search=10,
            ls_c=1e-4)


def listed():
    return [
        # the smallest call: the tangent of a 4^3 block, dominated by launches
        dict(name="assemble_fp64_4", kind="assemble", N=4, prec="fp64", bc=True, jitter=0.0,
             sigma=0.0, nu=0.3),
        # an odd, jittered, mid-size tangent in FP32 with the Dirichlet rows
        # eliminated: one mixed Newton iteration's assembly
        dict(name="assemble_mixed_33", kind="assemble", N=33, prec="mixed", bc=True, jitter=0.15,
             sigma=0.3, nu=0.3),
        # the assembly workload (log-normal mu, sinusoidal u): 12.6 M tets
        dict(name="assemble_fp64_128", kind="assemble", N=128, prec="fp64", bc=False, jitter=0.0,
             sigma=0.3, nu=0.3),
        # a line-search trial point of the 64^3 block
        dict(name="residual_64", kind="residual", N=64, jitter=0.15, sigma=0.3, nu=0.3),
        # independent tets in one batch (not a multiple of any tile)
        dict(name="elements_200k", kind="elements", n=200003, nu=0.3),
        # factorization and one apply on an odd mesh: the preconditioner alone
        dict(name="ilu_apply_31", kind="ilu_apply", N=31, jitter=0.0, sigma=0.3, nu=0.3),
        # pcg_solve_ilu0 as a user calls it: factorize, solve to 1e-12
        dict(name="pcg_fp64_48", kind="pcg", N=48, jitter=0.1, sigma=0.3, nu=0.3),
        # the host-array drop-in on a 2-D five-point diffusion matrix
        dict(name="csr_pcg_150", kind="csr_pcg", g=150, sigma=0.5),
        # a load step of the 8^3 parity block (with a per-element modulus):
        # many small launches
        dict(name="newton_fp64_8", kind="newton", N=8, prec="fp64", jitter=0.0, sigma=0.3, nu=0.3,
             uz=-0.1, n_steps=5),
        # a load step of the benchmark's 64^3 block with its mixed settings
        dict(name="newton_mixed_64", kind="newton", N=64, prec="mixed", jitter=0.15, sigma=0.3,
             nu=0.3, uz=-0.2, n_steps=10),
        # the backward direction: material gradients on the 32^3 block
        dict(name="adjoint_mixed_32", kind="adjoint", N=32, prec="mixed", jitter=0.0, sigma=0.3,
             nu=0.3),
        # the engine's state update after a Newton iteration, 48^3
        dict(name="states_48", kind="states", N=48, sigma=0.3, nu=0.3),
    ]


def draw(rng):
    """A case of the same kinds with sizes over the whole range (odd and
    ragged ones among them)."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["assemble", "assemble", "residual", "elements", "ilu_apply", "pcg",
                       "csr_pcg", "newton", "newton", "adjoint", "states"])
    jitter = rng.choice([0.0, 0.05, 0.1, 0.15])
    sigma = rng.choice([0.0, 0.2, 0.3])
    nu = round(rng.uniform(0.2, 0.35), 3)
    c = dict(kind=kind, nu=nu, sigma=sigma)
    if kind == "assemble":
        c.update(N=size(4, 128), prec=rng.choice(["fp64", "mixed"]), bc=rng.random() < 0.5,
                 jitter=jitter)
    elif kind == "residual":
        c.update(N=size(4, 128), jitter=jitter)
    elif kind == "elements":
        c = dict(kind=kind, n=size(300, 400000), nu=nu)
    elif kind == "ilu_apply":
        c.update(N=size(4, 64), jitter=jitter)
    elif kind == "pcg":
        c.update(N=size(6, 48), jitter=jitter)
    elif kind == "csr_pcg":
        c = dict(kind=kind, g=size(12, 150), sigma=rng.choice([0.0, 0.3, 0.5]))
    elif kind == "newton":
        if rng.random() < 0.5:
            c.update(N=size(4, 10), prec="fp64", uz=-0.1, n_steps=5)
        else:
            c.update(N=size(8, 56), prec="mixed", uz=-0.2, n_steps=10)
        c.update(jitter=jitter, sigma=sigma or 0.2)
    elif kind == "adjoint":
        c.update(N=size(8, 32), prec="mixed", jitter=jitter)
    else:
        c.update(N=size(6, 64))
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _cube(N):
    """the undeformed cube: (xyz, conn, stored volumes)"""
    xyz, conn = F.unit_cube(N)
    return xyz, conn, configs.tet_volumes(xyz, conn)


def _mesh(case, seed):
    """(xyz, conn, stored volumes, per-element E or None) of the case's block"""
    xyz, conn, vol = _cube(case["N"])
    if case.get("jitter"):
        xyz = configs.jitter_interior(xyz, case["N"], case["jitter"], 2 * seed + 1)
    E = None
    if case.get("sigma"):
        E = configs.lognormal_E(conn.size // 4, case["sigma"], 2 * seed, case["nu"])
    return xyz, conn, vol, E


def _bc(case, xyz):
    # Dirichlet faces by the undeformed coordinates (jitter moves interior nodes only)
    return configs.clamp_top_bc(xyz, case.get("uz", -0.1))


def _field(xyz, seed, amp=0.05):
    """the assembly workload's sinusoidal displacement with seeded phases"""
    ph = np.random.default_rng(seed).uniform(0.0, 2.0 * np.pi, size=(3, 3))
    x, y, z = xyz[0::3], xyz[1::3], xyz[2::3]
    u = np.empty_like(xyz)
    for c in range(3):
        u[c::3] = amp * (np.sin(2 * np.pi * x + ph[c, 0]) * np.sin(2 * np.pi * y + ph[c, 1]) *
                         np.sin(2 * np.pi * z + ph[c, 2]))
    return u


def _loaded_state(xyz, seed):
    """a smooth state of the compressed block after its first load steps:
    u_z linear in z (clamped bottom, top at -0.02), sides bulging, with a
    small seeded ripple; bulge and ripple vanish on both faces"""
    u = _field(xyz, seed, amp=0.001)
    z = xyz[2::3]
    for c in range(3):
        if c < 2:
            u[c::3] += 0.006 * (xyz[c::3] - 0.5)
        u[c::3] *= np.sin(np.pi * z)
    u[2::3] += -0.02 * z
    return u


def _rhs(case, seed, mask):
    b = np.random.default_rng(seed).standard_normal(mask.size)
    b[mask == 1] = 0.0
    return b


def _diffusion(case, seed):
    """five-point diffusion matrix on a g x g grid, log-normal edge
    conductivities, Dirichlet surroundings: (row_ptr, col_idx, val, b)"""
    g = case["g"]
    rng = np.random.default_rng(seed)
    kx = np.exp(case["sigma"] * rng.standard_normal((g, g + 1)))
    ky = np.exp(case["sigma"] * rng.standard_normal((g + 1, g)))
    b = rng.standard_normal(g * g)
    idx = np.arange(g * g).reshape(g, g)
    diag = kx[:, :-1] + kx[:, 1:] + ky[:-1] + ky[1:]
    # neighbours in ascending column order: north, west, self, east, south
    cols = np.full((g, g, 5), -1, np.int64)
    vals = np.zeros((g, g, 5))
    cols[1:, :, 0], vals[1:, :, 0] = idx[:-1], -ky[1:-1]
    cols[:, 1:, 1], vals[:, 1:, 1] = idx[:, :-1], -kx[:, 1:-1]
    cols[:, :, 2], vals[:, :, 2] = idx, diag
    cols[:, :-1, 3], vals[:, :-1, 3] = idx[:, 1:], -kx[:, 1:-1]
    cols[:-1, :, 4], vals[:-1, :, 4] = idx[1:], -ky[1:-1]
    cols, vals = cols.reshape(-1, 5), vals.reshape(-1, 5)
    keep = cols >= 0
    rp = np.zeros(g * g + 1, np.uint32)
    rp[1:] = np.cumsum(keep.sum(1))
    return rp, cols[keep].astype(np.uint32), vals[keep], b


def _batch(case, seed):
    """independent well-shaped tets: a unit corner tet of random size and
    orientation-preserving distortion, displaced by a few percent"""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["n"]

    def normal(*s):
        return torch.randn(*s, generator=g, device="cuda", dtype=torch.float64)

    ref = torch.tensor([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]], device="cuda",
                       dtype=torch.float64)
    h = 0.05 * torch.exp(0.3 * normal(n, 1, 1))
    x = h * (ref + 0.08 * normal(n, 4, 3)) + normal(n, 1, 3)
    u = 0.03 * h * normal(n, 4, 3)
    E = torch.exp(0.3 * normal(n))
    return x.reshape(n, 12).contiguous(), u.reshape(n, 12).contiguous(), E


def prepare(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda:0")
    s = {"case": case}

    def cu(a):
        return torch.as_tensor(a, device=dev)

    if kind == "csr_pcg":
        s["ctx"] = F.Context(0)
        s["system"] = _diffusion(case, seed)
        return s
    if kind == "elements":
        s["ctx"] = F.Context(0)
        s["x"], s["u"], s["E"] = _batch(case, seed)
        return s
    xyz, conn, vol, E = _mesh(case, seed)
    mask, val = _bc(case, xyz)
    ctx = F.Context(0)
    ctx.set_mesh(xyz, conn, vol)
    ctx.set_material(1.0, case["nu"], E)
    ctx.set_bc(mask, val)
    s["ctx"] = ctx
    n = ctx.n_dofs
    if kind == "assemble":
        s["u"] = cu(_field(xyz, seed))
        s["K"] = torch.zeros(ctx.nnz, device=dev,
                             dtype=torch.float64 if case["prec"] == "fp64" else torch.float32)
        s["f"] = torch.zeros(n, dtype=torch.float64, device=dev)
    elif kind == "residual":
        s["u"] = cu(_field(xyz, seed))
        s["f"] = torch.zeros(n, dtype=torch.float64, device=dev)
    elif kind in ("ilu_apply", "pcg"):
        ctx.assemble_into_context(cu(_loaded_state(xyz, seed)), apply_bc=True)
        s["b"] = cu(_rhs(case, seed + 1, mask))
    elif kind == "newton":
        s["u"] = torch.zeros(n, dtype=torch.float64, device=dev)
        s["cfg"] = dict(FP64 if case["prec"] == "fp64" else MIXED, prec=PREC[case["prec"]])
    elif kind == "adjoint":
        s["u"] = cu(_loaded_state(xyz, seed))
        g = np.zeros(n)
        sel = configs.top_face_xy_dofs(xyz)
        g[sel] = np.random.default_rng(seed + 1).standard_normal(sel.size)
        s["g"] = cu(g)
    elif kind == "states":
        s["u"] = cu(_field(xyz, seed, amp=0.02))
        s["F"] = torch.eye(3, dtype=torch.float64, device=dev).reshape(1, 9).repeat(
            ctx.n_elems, 1).contiguous()
        s["stress"] = torch.zeros(ctx.n_elems, 6, dtype=torch.float64, device=dev)
    else:
        raise ValueError(kind)
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "assemble":
        return ctx.assemble(s["u"], prec=PREC[case["prec"]], apply_bc=case["bc"], K=s["K"],
                            f=s["f"])
    if kind == "residual":
        return ctx.residual(s["u"], f=s["f"])
    if kind == "elements":
        return ctx.elements(s["x"], s["u"], s["E"], case["nu"])
    if kind == "ilu_apply":
        ctx.ilu0()
        return ctx.ilu0_apply(s["b"])
    if kind == "pcg":
        ctx.ilu0()
        return ctx.pcg(s["b"], tol=1e-12, max_iter=5000)[0]
    if kind == "csr_pcg":
        return ctx.csr_pcg_ilu0(*s["system"], tol=1e-12, max_iter=5000)[0]
    if kind == "newton":
        u = s["u"].clone()
        ctx.newton_step_cfg(u, 1.0 / case["n_steps"], **s["cfg"])
        return u
    if kind == "adjoint":
        return ctx.adjoint(s["u"], s["g"], tol=1e-11, inner_tol=0.1, prec=PREC[case["prec"]],
                           want_w=True)[:3]
    F_sl3, stress, _ = ctx.element_states(s["u"], s["F"], s["stress"])
    return F_sl3, stress


# ---------------------------------------------------------------------------
# the bytes and operations a pass cannot do without
# ---------------------------------------------------------------------------
def _sizes(N):
    """nodes, tets, node-neighbour entries (each node its own neighbour)"""
    nn = (N + 1) ** 3
    # edges of the split: three lattice directions, and face diagonals (the
    # two hexes at an interior face cut it along different diagonals)
    edges = 3 * N * (N + 1) ** 2 + 6 * N ** 3 + N * N
    return nn, 6 * N ** 3, nn + 2 * edges


def work(case):
    kind = case["kind"]
    if kind == "elements":
        n = case["n"]
        return {"bytes": 8 * n * (12 + 12 + 1 + 144 + 12), "flops": 1200 * n}
    if kind == "csr_pcg":
        g = case["g"]
        n, nnz = g * g, 5 * g * g - 4 * g
        # read once: the matrix, b, x; the iterations' operations (about 1.2 g of them)
        return {"bytes": 12 * nnz + 4 * (n + 1) + 8 * 3 * n, "flops": 1.2 * g * (4 * nnz + 10 * n)}
    nn, ne, entries = _sizes(case["N"])
    n, nnz = 3 * nn, 9 * entries
    mat = 8 * ne if case.get("sigma") else 0
    mesh = 16 * ne + mat + 24 * nn + 8 * n  # conn, E, xyz, u
    if kind == "assemble":
        w = 8 if case["prec"] == "fp64" else 4
        return {"bytes": mesh + w * nnz + 8 * n, "flops": 900 * ne}
    if kind == "residual":
        return {"bytes": mesh + 8 * n, "flops": 250 * ne}
    if kind == "states":
        return {"bytes": mesh + 120 * ne, "flops": 300 * ne}
    # per lower-upper pair of a row's blocks: about 9 steps of 3x3 updates per node
    ilu_flops = 54.0 * 9 * entries
    if kind == "ilu_apply":
        return {"bytes": 8 * (2 * nnz + 2 * n) + 4 * entries, "flops": ilu_flops + 2 * nnz}
    if kind == "pcg":
        its = 5.5 * case["N"] ** 0.9
        return {"bytes": 8 * (2 * nnz + 2 * n) + 4 * entries,
                "flops": ilu_flops + its * (4 * nnz + 10 * n)}
    if kind == "newton":
        if case["prec"] == "fp64":
            solves, its = 60, 60 * 5.5 * case["N"] ** 0.9
        else:
            solves, its = 75, 60.0 + 18.0 * case["N"]
        return {"bytes": mesh + 8 * n + n, "flops": solves * 1200 * ne + its * (4 * nnz + 10 * n)}
    sweeps = 25
    return {"bytes": mesh + 8 * 3 * n + 16 * ne,
            "flops": sweeps * (400 * ne + 2.0 * case["N"] * (4 * nnz + 10 * n))}


# ---------------------------------------------------------------------------
# the same outputs from plain FP64 torch
# ---------------------------------------------------------------------------
class _Tets:
    """Element quantities of a set of tets in FP64 torch: shape gradients
    g_a, F = I + sum u_a (x) g_a, J, the Mandel stress M = mu (C - I) + lam
    ln J I, forces vol M g_a and the tangent the engine uses."""

    def __init__(self, x, u, mu, lam, nu):
        e1 = x[:, 1:] - x[:, :1]            # rows x_a - x_0
        inv = torch.linalg.inv(e1)           # grad N_a = column a of inv
        self.vol = torch.linalg.det(e1).abs() / 6.0
        g = torch.empty_like(x)
        g[:, 1:] = inv.transpose(1, 2)
        g[:, 0] = -g[:, 1:].sum(1)
        self.g = g
        eye = torch.eye(3, dtype=x.dtype, device=x.device)
        self.F = eye + torch.einsum("eai,eaj->eij", u, g)
        self.J = torch.linalg.det(self.F)
        self.mu, self.lam, self.nu = mu, lam, nu
        C = self.F.transpose(1, 2) @ self.F
        self.CmI = C - eye
        self.lnJ = torch.log(self.J)
        self.M = mu[:, None, None] * self.CmI + (lam * self.lnJ)[:, None, None] * eye

    def forces(self):
        return self.vol[:, None, None] * torch.einsum("eij,eaj->eai", self.M, self.g)

    def tangent(self):
        """[e, 4, 3, 4, 3]"""
        mu, lam = self.mu, self.lam
        bulk = lam + 2.0 * mu / 3.0
        a = 2.0 * mu + bulk + lam / (self.J * max(1.0 - 2.0 * self.nu, 0.1))
        b = bulk - 2.0 * mu / 3.0 - 2.0 * lam * self.lnJ / (3.0 * self.J)
        v = self.vol
        t = torch.einsum("eip,ejq->eipjq", self.g, self.g)
        K = (v * b)[:, None, None, None, None] * t + \
            (v * mu)[:, None, None, None, None] * t.permute(0, 1, 4, 3, 2)
        dot = torch.einsum("eip,ejp->eij", self.g, self.g)
        geo = torch.einsum("eip,epq,ejq->eij", self.g, self.M, self.g)
        for p in range(3):
            tpp = t[:, :, p, :, p]
            w = v[:, None, None]
            K[:, :, p, :, p] = w * (a[:, None, None] * tpp + mu[:, None, None] * (dot - tpp) + geo)
        return K

    def exact_tangent(self):
        """derivative of forces() with respect to the 12 displacements:
        dM = mu (V^T F + F^T V) + lam tr(F^-1 V) I for V = e_q (x) g_b"""
        Fi = torch.linalg.inv(self.F)
        # (V^T F)_ij = g_b,i F_q,j
        gF = torch.einsum("ebi,eqj->ebqij", self.g, self.F)
        dM = self.mu[:, None, None, None, None] * (gF + gF.transpose(3, 4))
        tr = torch.einsum("eiq,ebi->ebq", Fi, self.g)
        eye = torch.eye(3, dtype=self.F.dtype, device=self.F.device)
        dM = dM + (self.lam[:, None, None] * tr)[..., None, None] * eye
        return self.vol[:, None, None, None, None] * torch.einsum("ebqij,eaj->eaibq", dM, self.g)


class _Block:
    """the active tets of a case's mesh on the GPU, for the exact values"""

    def __init__(self, case, seed):
        xyz, conn, vol, E = _mesh(case, seed)
        self.xyz_h = xyz
        dev = "cuda:0"
        self.ne = conn.size // 4
        self.active = torch.as_tensor(vol >= 1e-30, device=dev)
        self.conn_all = torch.as_tensor(conn.astype(np.int64), device=dev).view(-1, 4)
        self.conn = self.conn_all[self.active]
        self.xyz = torch.as_tensor(xyz, device=dev).view(-1, 3)
        E = torch.ones(self.ne, dtype=torch.float64, device=dev) if E is None else \
            torch.as_tensor(E, device=dev)
        self.nu = nu = case["nu"]
        self.mu_all = E / (2.0 * (1.0 + nu))
        self.lam_all = E * nu / ((1.0 + nu) * (1.0 - 2.0 * nu))
        self.mu, self.lam = self.mu_all[self.active], self.lam_all[self.active]
        self.n = xyz.size
        mask, val = _bc(case, xyz)
        self.mask_h = mask
        self.free = torch.as_tensor(mask == 0, device=dev)
        self.val = torch.as_tensor(val, device=dev)
        self.dofs = (3 * self.conn[:, :, None] + torch.arange(3, device=dev)).reshape(-1, 12)

    def cu(self, a):
        return torch.as_tensor(a, device=self.xyz.device)

    def tets(self, u, part=slice(None)):
        c = self.conn[part]
        return _Tets(self.xyz[c], u.view(-1, 3)[c], self.mu[part], self.lam[part], self.nu)

    def parts(self):
        n = self.conn.shape[0]
        return [slice(b, min(n, b + (1 << 19))) for b in range(0, n, 1 << 19)]

    def force(self, u):
        f = torch.zeros_like(u)
        for p in self.parts():
            f.index_add_(0, self.dofs[p].reshape(-1), self.tets(u, p).forces().reshape(-1))
        return f

    def element_matrices(self, u, exact=False):
        return torch.cat([(t.exact_tangent() if exact else t.tangent()).reshape(-1, 12, 12)
                          for t in (self.tets(u, p) for p in self.parts())])

    def product(self, Ke, v):
        y = torch.zeros_like(v)
        y.index_add_(0, self.dofs.reshape(-1),
                     torch.bmm(Ke, v[self.dofs][:, :, None]).reshape(-1))
        return y

    def diagonal(self, Ke):
        d = torch.zeros(self.n, dtype=torch.float64, device=Ke.device)
        d.index_add_(0, self.dofs.reshape(-1),
                     torch.diagonal(Ke, dim1=1, dim2=2).reshape(-1))
        return torch.where(self.free, d, torch.ones_like(d))

    def solve(self, Ke, b, tol, max_iter=20000):
        """Jacobi-PCG on the free DOFs"""
        di = 1.0 / self.diagonal(Ke)
        b = torch.where(self.free, b, torch.zeros_like(b))
        x = torch.zeros_like(b)
        r, stop = b.clone(), tol * float(b.norm())
        z = di * r
        p, rz = z.clone(), torch.dot(r, z)
        for it in range(max_iter):
            q = torch.where(self.free, self.product(Ke, p), torch.zeros_like(p))
            alpha = rz / torch.dot(p, q)
            x += alpha * p
            r -= alpha * q
            if it % 8 == 7 and float(r.norm()) <= stop:
                break
            z = di * r
            rz, old = torch.dot(r, z), rz
            p = z + (rz / old) * p
        return x

    def csr(self):
        """(neighbour-entry keys n * Nn + m ascending, row offsets, positions)"""
        nn = self.n // 3
        c = self.conn_all
        keys = torch.empty(0, dtype=torch.int64, device=c.device)
        for b in range(0, c.shape[0], 1 << 20):
            k = (c[b:b + (1 << 20), :, None] * nn + c[b:b + (1 << 20), None, :]).reshape(-1)
            keys = torch.unique(torch.cat([keys, torch.unique(k)]))
        ptr = torch.searchsorted(keys, nn * torch.arange(nn + 1, device=c.device))
        return keys, ptr

    def matrix(self, u, bc):
        """the scalar CSR values: row 3n+p holds 3 columns per neighbour of n"""
        nn = self.n // 3
        keys, ptr = self.csr()
        K = torch.zeros(9 * keys.numel(), dtype=torch.float64, device=u.device)
        three = torch.arange(3, device=u.device)
        for part in self.parts():
            c = self.conn[part]
            k = torch.searchsorted(keys, (c[:, :, None] * nn + c[:, None, :]))
            k -= ptr[c][:, :, None]          # position in the row node's list
            deg = ptr[c + 1] - ptr[c]
            slot = (9 * ptr[c][:, :, None, None, None] +
                    3 * three[None, None, :, None, None] * deg[:, :, None, None, None] +
                    3 * k[:, :, None, :, None] + three[None, None, None, None, :])
            K.index_add_(0, slot.reshape(-1), self.tets(u, part).tangent().reshape(-1))
        if bc:
            row_n, col_n = keys // nn, keys % nn
            fixed = ~self.free.view(-1, 3)
            j = torch.arange(keys.numel(), device=u.device) - ptr[row_n]
            deg = ptr[row_n + 1] - ptr[row_n]
            for p in range(3):
                for q in range(3):
                    at = 9 * ptr[row_n] + 3 * p * deg + 3 * j + q
                    cut = fixed[row_n, p] | fixed[col_n, q]
                    one = ((row_n == col_n) & (p == q)).to(torch.float64)
                    K[at] = torch.where(cut, one, K[at])
        return K


def _exact_newton(B, frac):
    """equilibrium of the load step: the engine's tangent in a Newton
    iteration with loose inner solves, to a residual of 1e-13"""
    u = torch.zeros(B.n, dtype=torch.float64, device="cuda:0")
    v = torch.where(B.free, torch.zeros_like(u), frac * B.val)
    Ke = B.element_matrices(u)
    R = torch.where(B.free, -B.force(u) - B.product(Ke, v), torch.zeros_like(u))
    r0 = float(R.norm())
    u = u + v + B.solve(Ke, R, 1e-5)
    last = math.inf
    for _ in range(200):
        R = torch.where(B.free, -B.force(u), torch.zeros_like(u))
        rn = float(R.norm())
        if rn < 1e-13 * r0 or (rn < 1e-11 * r0 and rn > 0.9 * last):
            break
        last = rn
        u = u + B.solve(B.element_matrices(u), R, 0.05)
    return u


def _exact_adjoint(B, u, g):
    """K^T w = g on the free DOFs (K: derivative of the force) by BiCGStab
    with restarts, then the parameter derivatives of -w . f"""
    KT = B.element_matrices(u, exact=True).transpose(1, 2).contiguous()
    di = 1.0 / B.diagonal(KT)
    zero = torch.zeros_like(g)

    def A(v):
        return torch.where(B.free, B.product(KT, v), zero)

    g = torch.where(B.free, g, zero)
    w, gn = zero.clone(), float(g.norm())
    for _ in range(12):
        r = g - A(w)
        if float(r.norm()) <= 1e-14 * gn:
            break
        stop = 1e-4 * float(r.norm())
        rh, p, x = r.clone(), r.clone(), zero.clone()
        rho = torch.dot(rh, r)
        for it in range(3000):
            ph = di * p
            q = A(ph)
            alpha = rho / torch.dot(rh, q)
            s = r - alpha * q
            sh = di * s
            t = A(sh)
            om = torch.dot(t, s) / torch.dot(t, t)
            x += alpha * ph + om * sh
            r = s - om * t
            if it % 4 == 3 and float(r.norm()) <= stop:
                break
            rho, old = torch.dot(rh, r), rho
            p = r + (rho / old) * (alpha / om) * (p - om * q)
        w = w + x
    T = B.tets(u)
    L = torch.einsum("eai,eaj->eij", w.view(-1, 3)[B.conn], T.g)
    gm = torch.zeros(B.ne, dtype=torch.float64, device=g.device)
    gl = torch.zeros_like(gm)
    gm[B.active] = -T.vol * (T.CmI * L).sum((1, 2))
    gl[B.active] = -T.vol * T.lnJ * torch.diagonal(L, dim1=1, dim2=2).sum(1)
    return gm, gl, w


def exact(case, seed):
    kind = case["kind"]
    if kind == "elements":
        x, u, E = _batch(case, seed)
        nu = case["nu"]
        out_K, out_f = [], []
        for b in range(0, case["n"], 1 << 17):
            e = E[b:b + (1 << 17)]
            T = _Tets(x[b:b + (1 << 17)].view(-1, 4, 3), u[b:b + (1 << 17)].view(-1, 4, 3),
                      e / (2.0 * (1.0 + nu)), e * nu / ((1.0 + nu) * (1.0 - 2.0 * nu)), nu)
            out_K.append(T.tangent().reshape(-1, 144))
            out_f.append(T.forces().reshape(-1, 12))
        return torch.cat(out_K), torch.cat(out_f)
    if kind == "csr_pcg":
        rp, ci, val, b = _diffusion(case, seed)
        A = torch.sparse_csr_tensor(torch.as_tensor(rp.astype(np.int64)),
                                    torch.as_tensor(ci.astype(np.int64)), torch.as_tensor(val),
                                    size=(b.size, b.size)).to("cuda:0")
        bb = torch.as_tensor(b, device="cuda:0")
        x = torch.zeros_like(bb)
        for _ in range(3):  # CG, restarted on the true residual
            r = bb - A @ x
            p, rr = r.clone(), torch.dot(r, r)
            d = torch.zeros_like(x)
            stop = 1e-22 * float(rr)
            for it in range(20000):
                q = A @ p
                a = rr / torch.dot(p, q)
                d += a * p
                r -= a * q
                rr, old = torch.dot(r, r), rr
                if it % 16 == 15 and float(rr) <= stop:
                    break
                p = r + (rr / old) * p
            x = x + d
        return x.cpu().numpy()
    if kind == "ilu_apply":
        return None  # ILU(0) is sequential over rows: no plain torch form of it is quick
    if kind == "newton" and case["N"] > 32:
        return None  # nested Newton-CG without a good preconditioner: over 20 s
    B = _Block(case, seed)
    if kind == "assemble":
        u = B.cu(_field(B.xyz_h, seed))
        return B.matrix(u, case["bc"]), B.force(u)
    if kind == "residual":
        return B.force(B.cu(_field(B.xyz_h, seed)))
    if kind == "states":
        # exp(log F) rescaled to det 1 is F / cbrt(det F); stress of that F,
        # whose ln J is zero
        u = B.cu(_field(B.xyz_h, seed, amp=0.02))
        T = B.tets(u)
        Fs = T.F / (T.J ** (1.0 / 3.0))[:, None, None]
        eye = torch.eye(3, dtype=torch.float64, device=u.device)
        M = T.mu[:, None, None] * (Fs.transpose(1, 2) @ Fs - eye)
        F_all = eye.reshape(1, 9).repeat(B.ne, 1)
        S_all = torch.zeros(B.ne, 6, dtype=torch.float64, device=u.device)
        F_all[B.active] = Fs.reshape(-1, 9)
        r2 = math.sqrt(2.0)
        S_all[B.active] = torch.stack([M[:, 0, 0], M[:, 1, 1], M[:, 2, 2], r2 * M[:, 0, 1],
                                       r2 * M[:, 0, 2], r2 * M[:, 1, 2]], 1)
        return F_all, S_all
    if kind == "pcg":
        Ke = B.element_matrices(B.cu(_loaded_state(B.xyz_h, seed)))
        b = B.cu(_rhs(case, seed + 1, B.mask_h))
        x = B.solve(Ke, b, 1e-13)
        r = torch.where(B.free, b - B.product(Ke, x), torch.zeros_like(b))
        return x + B.solve(Ke, r, 1e-4)
    if kind == "newton":
        return _exact_newton(B, 1.0 / case["n_steps"])
    u = B.cu(_loaded_state(B.xyz_h, seed))
    g = np.zeros(B.n)
    sel = configs.top_face_xy_dofs(B.xyz_h)
    g[sel] = np.random.default_rng(seed + 1).standard_normal(sel.size)
    return _exact_adjoint(B, u, B.cu(g))
