"""Performance cases: what a program that uses this framework has it do.

Each case is a dict of plain values; prepare() makes the operators and inputs that a user's
program holds, run() makes one pass through the public entry points of `pmg`, work() counts
what the pass cannot do without, and exact() gives the same outputs in 64 bits from plain
torch (its own tables, numbering, geometry and operators).

Kinds of cases:
  vmult    one application of a continuous Q_p Laplace operator (LaplaceOperator.vmult)
  dg       one application of the DG-SIPG operator (DGLaplaceOperator.vmult)
  smooth   Chebyshev pre-smoothing from zero and post-smoothing (Chebyshev.vmult, .step)
  transfer restriction and prolongation between two levels (Transfer)
  vcycle   one multigrid V-cycle on an FP64 residual (VCycleMultigrid.vmult)
  solve    a whole multigrid-preconditioned CG solve (Hierarchy.solve)
  adjoint  the gradient of a misfit with respect to the coefficient (AdjointPoisson.gradient)
Meshes are boxes of coarse cells (cx, cy, cz) refined `refine` times; "geometry" is "affine"
(axis-aligned cells), "kappa" (affine cells, coefficient at every quadrature point) or
"deformed" (the sine-deformed cube with a full geometry tensor at every quadrature point).
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (os.path.join(_ROOT, "portable-multigrid_b200"), _ROOT):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import pmg  # noqa: E402
from pmg.adjoint import AdjointPoisson, fourier_field  # noqa: E402

DEV = 0


def _box(coarse, refine):
    return {"cx": coarse[0], "cy": coarse[1], "cz": coarse[2], "refine": refine}


def listed():
    return [
        # the smallest call: the operator of the plain Q2 h-multigrid example on its finest mesh
        # (16^3 affine cells, 35,937 DoFs), where launches and latency count
        {"name": "vmult_q2_f64_affine_16", "kind": "vmult", "degree": 2, "dtype": "f64", "geometry": "affine",
         **_box((2, 2, 2), 3)},
        # an odd mesh: 3 x 5 x 7 coarse cells refined twice, deformed, Q3 (186,325 DoFs)
        {"name": "vmult_q3_f64_deformed_12x20x28", "kind": "vmult", "degree": 3, "dtype": "f64",
         "geometry": "deformed", **_box((3, 5, 7), 2)},
        # the single-precision operator of the operator benchmark in the middle of its refinement sweep
        {"name": "vmult_q4_f32_deformed_64", "kind": "vmult", "degree": 4, "dtype": "f32", "geometry": "deformed",
         **_box((1, 1, 1), 6)},
        # the headline operator benchmark at its largest size: 135,005,697 DoFs in double precision
        {"name": "vmult_q4_f64_deformed_128", "kind": "vmult", "degree": 4, "dtype": "f64", "geometry": "deformed",
         **_box((1, 1, 1), 7)},
        # the finest level of the variable-coefficient problem (Q6, 48^3 cells, 24.1M DoFs) in the precision of
        # the outer CG
        {"name": "vmult_q6_f64_kappa_48", "kind": "vmult", "degree": 6, "dtype": "f64", "geometry": "kappa",
         **_box((3, 3, 3), 4)},
        # the DG operator (Q3, 64^3 cells, 16.8M DoFs) in the precision of the V-cycle
        {"name": "dg_q3_f32_64", "kind": "dg", "degree": 3, "dtype": "f32", **_box((1, 1, 1), 6)},
        # smoothing as every level above the coarsest does it, on the doubling mesh of the reference's runs
        # (2 x 2 x 1 coarse cells refined five times, Q4, 8.5M DoFs)
        {"name": "smooth_q4_f32_affine_64x64x32", "kind": "smooth", "degree": 4, "dtype": "f32", "geometry": "affine",
         "cheb": 5, **_box((2, 2, 1), 5)},
        # the p-transfer of the same runs, both directions
        {"name": "transfer_q4_q2_f32_64x64x32", "kind": "transfer", "degree": 4, "coarse_degree": 2, "dtype": "f32",
         **_box((2, 2, 1), 5)},
        # one single-precision V-cycle (Q4, p 4-3-2-1 and Q1 h-levels, 32^3 cells, 2.1M DoFs), the preconditioner
        # of every CG iteration: a few large levels and many small ones
        {"name": "vcycle_q4_f32_32", "kind": "vcycle", "degree": 4, "dtype": "f32", "geometry": "affine", "cheb": 5,
         **_box((1, 1, 1), 5)},
        # a small whole solve: plain Q2 h-multigrid, double precision throughout, 16^3 cells
        {"name": "solve_q2_f64_plain_16", "kind": "solve", "degree": 2, "dtype": "f64", "geometry": "affine",
         "plain": True, "cheb": 3, **_box((2, 2, 2), 3)},
        # the whole mixed-precision solve of the variable-coefficient problem (p 6-3-2-1, FP32 V-cycle in FP64 CG)
        {"name": "solve_q6_f32_kappa_48", "kind": "solve", "degree": 6, "dtype": "f32", "geometry": "kappa",
         "plain": False, "cheb": 4, **_box((3, 3, 3), 4)},
        # the gradient of the inverse problem: coefficient load, forward and adjoint solve, per-point form
        {"name": "adjoint_q4_32", "kind": "adjoint", "degree": 4, **_box((1, 1, 1), 5)},
    ]


def draw(rng):
    """One more case of the same kinds: sizes spread over the logarithm of their range, every degree,
    precision and geometry, coarse meshes of any small shape."""
    kind = rng.choice(["vmult"] * 6 + ["dg"] * 2 + ["smooth"] * 2 + ["transfer"] * 2 + ["vcycle"] * 2 + ["solve", "adjoint"])

    def mesh(lo, hi, degree, min_refine=1):
        """About exp(U[log lo, log hi]) DoFs: a coarse box with 1 to 7 cells per direction, refined as needed;
        where a point smoother has to converge (min_refine 2) the cells are at most twice as long as wide."""
        cells = math.exp(rng.uniform(math.log(lo), math.log(hi))) / degree ** 3
        base = rng.randint(1, 3)
        c = [rng.randint(1, 7) if min_refine < 2 else base + rng.randint(0, 1) for _ in range(3)]
        r = max(min_refine, round(math.log(max(cells, 1.0) / (c[0] * c[1] * c[2]), 8)))
        while r > min_refine and c[0] * c[1] * c[2] * 8 ** r * degree ** 3 > 1.3 * hi:
            r -= 1
        while c[0] * c[1] * c[2] * 8 ** r * degree ** 3 > 1.3 * hi:
            c = [max(1, v // 2) for v in c]
        return _box(c, r)

    degree = rng.randint(1, 6)
    dtype = rng.choice(["f64", "f32"])
    if kind == "vmult":
        geometry = rng.choice(["affine", "deformed", "deformed", "kappa"])
        return {"kind": kind, "degree": degree, "dtype": dtype, "geometry": geometry, **mesh(2e4, 1.2e7, degree)}
    if kind == "dg":
        return {"kind": kind, "degree": degree, "dtype": dtype, **mesh(5e4, 1.2e7, degree + 1)}
    if kind == "smooth":
        return {"kind": kind, "degree": degree, "dtype": dtype, "geometry": rng.choice(["affine", "deformed", "kappa"]),
                "cheb": rng.randint(3, 6), **mesh(2e4, 1e7, degree)}
    if kind == "transfer":
        degree = max(2, degree)
        return {"kind": kind, "degree": degree, "coarse_degree": rng.choice([0] + list(range(1, degree))),
                "dtype": dtype, **mesh(2e4, 1e7, degree)}
    if kind == "vcycle":
        return {"kind": kind, "degree": degree, "dtype": dtype, "geometry": rng.choice(["affine", "deformed", "kappa"]),
                "cheb": rng.randint(3, 5), **mesh(2e4, 6e6, degree, 2)}
    if kind == "solve":
        return {"kind": kind, "degree": degree, "dtype": dtype, "geometry": "affine", "plain": False,
                "cheb": rng.randint(3, 5), **mesh(2e4, 5e6, degree, 2)}
    return {"kind": kind, "degree": rng.randint(2, 4), **mesh(2e4, 1.2e6, degree, 2)}


# ---- the user's program ---------------------------------------------------------------------


def _dt(case):
    return (pmg.F64, torch.float64) if case["dtype"] == "f64" else (pmg.F32, torch.float32)


def _pmg_box(case):
    return pmg.Box.make(coarse=(case["cx"], case["cy"], case["cz"]), refine=case["refine"],
                        deform=1 if case.get("geometry") == "deformed" else 0, amp=0.1)


def _op(case, mesh, degree, dt):
    geo = {"affine": pmg.GEOMETRY_AFFINE, "kappa": pmg.GEOMETRY_AFFINE,
           "deformed": pmg.GEOMETRY_FULL}[case.get("geometry", "affine")]
    kind = pmg.COEFF_KAPPA if case.get("geometry") == "kappa" else pmg.COEFF_NONE
    return pmg.LaplaceOperator(mesh, degree, dt, geo, kind, device=DEV)


def _uniform(n, seed, dtype):
    g = torch.Generator(device=f"cuda:{DEV}")
    g.manual_seed(int(seed))
    return (torch.rand(n, generator=g, dtype=torch.float64, device=f"cuda:{DEV}") * 2 - 1).to(dtype)


def _pseq(degree):
    """p-levels as the drivers use them: halving for the Q6 problem's 6-3-2-1, otherwise one by one."""
    return [6, 3, 2, 1] if degree == 6 else list(range(degree, 0, -1))


def _hierarchy(case):
    geo = pmg.GEOMETRY_FULL if case["geometry"] == "deformed" else pmg.GEOMETRY_AFFINE
    kind = pmg.COEFF_KAPPA if case["geometry"] == "kappa" else pmg.COEFF_NONE
    plain = case.get("plain", False)
    return pmg.Hierarchy(_pmg_box(case), [case["degree"]] if plain else _pseq(case["degree"]), mg_dtype=_dt(case)[0],
                         cheb_degree=case["cheb"], geometry=geo, coeff_kind=kind, device=DEV,
                         h_degree=case["degree"] if plain else 1)


def prepare(case, seed):
    torch.cuda.set_device(DEV)
    s = dict(case=case)
    kind = case["kind"]
    if kind in ("vmult", "dg", "smooth"):
        dt, tdt = _dt(case)
        s["mesh"] = pmg.Mesh(_pmg_box(case))
        if kind == "dg":
            s["op"] = pmg.DGLaplaceOperator(s["mesh"], case["degree"], dt, _penalty(case["degree"]), device=DEV)
        else:
            s["op"] = _op(case, s["mesh"], case["degree"], dt)
        s["src"] = _uniform(s["op"].m(), seed, tdt)
        s["dst"] = torch.empty_like(s["src"])
        if kind == "smooth":
            s["smoother"] = pmg.Chebyshev(s["op"], case["cheb"])
            s["smoother"].estimate()
    elif kind == "transfer":
        dt, tdt = _dt(case)
        if case["coarse_degree"]:
            s["mesh"] = pmg.Mesh(_pmg_box(case))
            s["coarse"] = _op(case, s["mesh"], case["coarse_degree"], dt)
        else:  # the geometric transfer from the next coarser mesh
            s["mesh"] = pmg.Mesh(_pmg_box(case))
            s["mesh_c"] = pmg.Mesh(_pmg_box(dict(case, refine=case["refine"] - 1)))
            s["coarse"] = _op(case, s["mesh_c"], case["degree"], dt)
        s["fine"] = _op(case, s["mesh"], case["degree"], dt)
        s["transfer"] = pmg.Transfer(s["coarse"], s["fine"])
        s["src_fine"] = _uniform(s["fine"].m(), seed, tdt)
        s["src_coarse"] = _uniform(s["coarse"].m(), seed + 1, tdt)
        s["dst_fine"] = torch.empty_like(s["src_fine"])
        s["dst_coarse"] = torch.empty_like(s["src_coarse"])
    elif kind in ("vcycle", "solve"):
        s["h"] = _hierarchy(case)
        s["h"].estimate()
        b = s["h"].fine64.assemble_rhs(0)
        s["b"] = b * (1.0 + 0.5 * _uniform(b.numel(), seed, torch.float64))
        s["x"] = torch.empty_like(s["b"])
    elif kind == "adjoint":
        s["problem"] = AdjointPoisson(_pmg_box(case), degree=case["degree"], device=DEV)
        xq = s["problem"].quadrature_points()
        s["u_d"] = s["problem"].solve(fourier_field(xq, seed=seed + 1))
        s["m"] = fourier_field(xq, seed=seed)
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind in ("vmult", "dg"):
        s["op"].vmult(s["dst"], s["src"])
        return s["dst"]
    if kind == "smooth":
        s["smoother"].vmult(s["dst"], s["src"])
        s["smoother"].step(s["dst"], s["src"])
        return s["dst"]
    if kind == "transfer":
        s["dst_coarse"].zero_()
        s["transfer"].restrict_and_add(s["dst_coarse"], s["src_fine"])
        s["dst_fine"].zero_()
        s["transfer"].prolongate_and_add(s["dst_fine"], s["src_coarse"])
        return s["dst_coarse"], s["dst_fine"]
    if kind == "vcycle":
        s["h"].mg.vmult(s["x"], s["b"])
        return s["x"]
    if kind == "solve":
        s["x"].zero_()
        s["h"].solve(s["b"], s["x"], reduce=1e-10)
        return s["x"]
    J, g, u = s["problem"].gradient(s["m"], s["u_d"])
    return J, g, u


# ---- what a pass cannot do without ----------------------------------------------------------


def _sizes(case, degree, refine=None):
    r = case["refine"] if refine is None else refine
    n = [case[k] << r for k in ("cx", "cy", "cz")]
    return n[0] * n[1] * n[2], (n[0] * degree + 1) * (n[1] * degree + 1) * (n[2] * degree + 1)


def _apply_work(case, degree, size, refine=None, geometry=None):
    """One operator application: source and result vectors, the index map, the stored geometry or
    coefficient per quadrature point; twelve 1D passes of N^4 multiply-adds and the point work per cell."""
    cells, dofs = _sizes(case, degree, refine)
    n = degree + 1
    geometry = geometry or case.get("geometry", "affine")
    per_point = {"affine": 0, "kappa": 1, "deformed": 6}[geometry]
    return (2 * size * dofs + cells * n ** 3 * (4 + per_point * size),
            cells * (24 * n ** 4 + (30 if geometry == "deformed" else 6) * n ** 3))


def _cycle_work(case, dtype_size):
    degree, cheb = case["degree"], case["cheb"]
    levels = [(degree if case.get("plain") else 1, r) for r in range(1, case["refine"] + 1)]
    if not case.get("plain"):
        levels += [(p, case["refine"]) for p in reversed(_pseq(degree)[:-1])]
    b = f = 0
    for p, r in levels:
        vb, vf = _apply_work(case, p, dtype_size, r)
        dofs = _sizes(case, p, r)[1]
        # pre-smoothing (cheb - 1 products), the residual, post-smoothing (cheb products); each step
        # reads the right-hand side and the diagonal beside its iterate
        b += 2 * cheb * (vb + 2 * dtype_size * dofs)
        f += 2 * cheb * vf
    return b, f


def work(case):
    kind = case["kind"]
    size = 4 if case.get("dtype") == "f32" else 8
    degree = case["degree"]
    if kind == "vmult":
        b, f = _apply_work(case, degree, size)
    elif kind == "dg":
        cells, _ = _sizes(case, degree)
        n = degree + 1
        b, f = 2 * size * cells * n ** 3, cells * (14 * n ** 4 + 6 * n ** 2 * (4 * n + 4 * n))
    elif kind == "smooth":
        vb, vf = _apply_work(case, degree, size)
        k = 2 * case["cheb"] - 1
        b, f = k * (vb + 2 * size * _sizes(case, degree)[1]), k * vf
    elif kind == "transfer":
        cd = case["coarse_degree"]
        cc, nc = _sizes(case, cd) if cd else _sizes(case, degree, case["refine"] - 1)
        nf = _sizes(case, degree)[1]
        a, n = (cd + 1, degree + 1) if cd else (degree + 1, 2 * degree + 1)
        b = 2 * (size * (nc + nf) + cc * (4 * (a ** 3 + n ** 3)))
        f = 2 * cc * 2 * (a ** 3 * n + a ** 2 * n ** 2 + a * n ** 3)
    elif kind == "vcycle":
        b, f = _cycle_work(case, size)
        b += 16 * _sizes(case, degree)[1]
    elif kind == "solve":
        its = 7
        cb, cf = _cycle_work(case, size)
        vb, vf = _apply_work(case, degree, 8)
        b, f = its * (cb + vb + 9 * 8 * _sizes(case, degree)[1]), its * (cf + vf)
    else:
        its = 2 * 11
        c = dict(case, cheb=4, geometry="kappa")
        cb, cf = _cycle_work(c, 4)
        vb, vf = _apply_work(c, degree, 8)
        b, f = its * (cb + vb + 9 * 8 * _sizes(case, degree)[1]), its * (cf + vf)
    return {"bytes": b, "flops": f}


# ---- the same outputs in 64 bits from plain torch -------------------------------------------


def _penalty(degree):
    return 2.0 * (degree + 1) ** 2


def _gll(p):
    """Gauss-Lobatto points on [0, 1]."""
    c = np.zeros(p + 1)
    c[p] = 1.0
    inner = np.polynomial.legendre.legroots(np.polynomial.legendre.legder(c)) if p > 1 else np.zeros(0)
    for _ in range(4):  # Newton steps on P_p'
        d1 = np.polynomial.legendre.legval(inner, np.polynomial.legendre.legder(c))
        d2 = np.polynomial.legendre.legval(inner, np.polynomial.legendre.legder(c, 2))
        inner = inner - d1 / np.where(d2 == 0, 1.0, d2)
    return 0.5 * (np.concatenate([[-1.0], inner, [1.0]]) + 1.0)


def _lagrange(nodes, x):
    """phi_i(x_q) and phi_i'(x_q) as [i][q]."""
    n = len(nodes)
    val, der = np.ones((n, len(x))), np.zeros((n, len(x)))
    for i in range(n):
        for m in range(n):
            if m != i:
                val[i] *= (x - nodes[m]) / (nodes[i] - nodes[m])
        for k in range(n):
            if k != i:
                t = np.full(len(x), 1.0 / (nodes[i] - nodes[k]))
                for m in range(n):
                    if m != i and m != k:
                        t *= (x - nodes[m]) / (nodes[i] - nodes[m])
                der[i] += t
    return val, der


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=f"cuda:{DEV}")


class _Space:
    """Tables, cells in Morton order and the first-visit numbering of FE_Q(p) on a box."""

    def __init__(self, case, degree, refine=None):
        r = case["refine"] if refine is None else refine
        coarse = (case["cx"], case["cy"], case["cz"])
        self.p, self.N = degree, degree + 1
        x, w = np.polynomial.legendre.leggauss(self.N)
        self.xg, self.wg = 0.5 * (x + 1.0), 0.5 * w
        self.xl = _gll(degree)
        S, SD = _lagrange(self.xl, self.xg)
        self.S, self.SD, self.W = _t(S), _t(SD), _t(self.wg)
        self.n = [c << r for c in coarse]
        self.h = [1.0 / n for n in self.n]
        dev = f"cuda:{DEV}"
        code = torch.arange(8 ** r, device=dev)
        loc = [sum(((code >> (3 * b + d)) & 1) << b for b in range(r)) if r else torch.zeros_like(code) for d in range(3)]
        tree = torch.arange(coarse[0] * coarse[1] * coarse[2], device=dev)
        t3 = [tree % coarse[0], (tree // coarse[0]) % coarse[1], tree // (coarse[0] * coarse[1])]
        self.xyz = torch.stack([((t3[d] << r)[:, None] + loc[d][None, :]).reshape(-1) for d in range(3)], 1)
        self.C = self.xyz.shape[0]
        self.chunk = max(1, (1 << 23) // self.N ** 3)

    def cells(self):
        for c0 in range(0, self.C, self.chunk):
            yield c0, min(self.C, c0 + self.chunk)

    def lattice(self, c0, c1):
        """Node-lattice index [cells, k, j, i] of the cells c0..c1."""
        L0, L1 = self.p * self.n[0] + 1, self.p * self.n[1] + 1
        a = torch.arange(self.N, device=self.xyz.device)
        x, y, z = (self.xyz[c0:c1, d, None] * self.p + a for d in range(3))
        return (z[:, :, None, None] * L1 + y[:, None, :, None]) * L0 + x[:, None, None, :]

    def number(self):
        """lattice -> DoF: nodes numbered at the first cell that holds them, x fastest inside the cell."""
        n_nodes = math.prod(self.p * n + 1 for n in self.n)
        n3 = self.N ** 3
        first = torch.full((n_nodes,), self.C * n3, dtype=torch.int64, device=self.xyz.device)
        for c0, c1 in self.cells():
            lat = self.lattice(c0, c1).reshape(-1)
            key = torch.arange(c0 * n3, c1 * n3, device=lat.device)
            first.scatter_reduce_(0, lat, key, "amin")
        flag = torch.zeros(self.C * n3, dtype=torch.bool, device=first.device)
        flag[first] = True
        rank = torch.cumsum(flag, 0, dtype=torch.int32)
        del flag
        self.dof = (rank[first] - 1).to(torch.int64)
        del rank, first
        g = [torch.arange(self.p * n + 1, device=self.dof.device) for n in self.n]
        edge = [(v == 0) | (v == self.p * n) for v, n in zip(g, self.n)]
        on = edge[2][:, None, None] | edge[1][None, :, None] | edge[0][None, None, :]
        self.constrained = torch.zeros(n_nodes, dtype=torch.bool, device=self.dof.device)
        self.constrained[self.dof] = on.reshape(-1)
        self.m = n_nodes
        return self

    def map(self, c0, c1):
        return self.dof[self.lattice(c0, c1)]


def _con(M, u, d):
    """Apply M[i][o] along direction d (0: x, the last axis) of u[cells, k, j, i]."""
    return torch.movedim(torch.tensordot(u, M, dims=([3 - d], [0])), -1, 3 - d)


def _kappa(x):
    s = torch.sin(2 * math.pi * x[0]) * torch.sin(2 * math.pi * x[1]) * torch.sin(2 * math.pi * x[2])
    return 1.0 + 0.9 * s


def _geometry(sp, case, c0, c1):
    """The symmetric tensor of each quadrature point as a 3 x 3 list of [cells, q2, q1, q0] (None: zero)."""
    w3 = sp.W[:, None, None] * sp.W[None, :, None] * sp.W[None, None, :]
    xl, xg = _t(sp.xl), _t(sp.xg)
    cc = sp.xyz[c0:c1].to(torch.float64)
    if case.get("geometry") != "deformed":
        vol = sp.h[0] * sp.h[1] * sp.h[2]
        f = w3[None] * vol
        if case.get("geometry") == "kappa":
            pts = [(cc[:, d, None] + xg[None, :]) * sp.h[d] for d in range(3)]
            f = f * _kappa([pts[0][:, None, None, :], pts[1][:, None, :, None], pts[2][:, :, None, None]])
        return [[f / sp.h[a] ** 2 if a == b else None for b in range(3)] for a in range(3)]
    pts = [(cc[:, d, None] + xl[None, :]) * sp.h[d] for d in range(3)]
    x, y, z = pts[0][:, None, None, :], pts[1][:, None, :, None], pts[2][:, :, None, None]
    s = 0.1 * torch.sin(math.pi * x) * torch.sin(math.pi * y) * torch.sin(math.pi * z)
    J = []
    for X in (x + s, y + s, z + s):
        J.append([_con(sp.SD if d == 2 else sp.S, _con(sp.SD if d == 1 else sp.S, _con(sp.SD if d == 0 else sp.S, X, 0), 1), 2)
                  for d in range(3)])
    adj = [[J[(b + 1) % 3][(a + 1) % 3] * J[(b + 2) % 3][(a + 2) % 3] - J[(b + 1) % 3][(a + 2) % 3] * J[(b + 2) % 3][(a + 1) % 3]
            for b in range(3)] for a in range(3)]  # det J^{-1}[a][b]
    det = sum(J[0][a] * adj[a][0] for a in range(3))
    f = w3[None] / det.abs()
    return [[f * sum(adj[a][k] * adj[b][k] for k in range(3)) for b in range(3)] for a in range(3)]


def _vmult64(sp, case, src, geo=None):
    """A src on FE_Q(p), Dirichlet rows the identity; geo: {first cell: tensor} kept between calls."""
    u = torch.where(sp.constrained, torch.zeros((), dtype=torch.float64, device=src.device), src)
    dst = torch.zeros_like(u)
    for c0, c1 in sp.cells():
        idx = sp.map(c0, c1)
        G = geo[c0] if geo is not None else _geometry(sp, case, c0, c1)
        e = u[idx]
        sx, dx = _con(sp.S, e, 0), _con(sp.SD, e, 0)
        sxy = _con(sp.S, sx, 1)
        g = [_con(sp.S, _con(sp.S, dx, 1), 2), _con(sp.S, _con(sp.SD, sx, 1), 2), _con(sp.SD, sxy, 2)]
        f = [sum(G[a][b] * g[b] for b in range(3) if G[a][b] is not None) for a in range(3)]
        St, Dt = sp.S.T, sp.SD.T
        o = _con(Dt, _con(St, _con(St, f[0], 2), 1), 0) + _con(St, _con(Dt, _con(St, f[1], 2), 1) + _con(St, _con(Dt, f[2], 2), 1), 0)
        dst.index_add_(0, idx.reshape(-1), o.reshape(-1))
    return torch.where(sp.constrained, src, dst)


def _diagonal64(sp, case):
    out = torch.zeros(sp.m, dtype=torch.float64, device=sp.dof.device)
    t = (sp.S, sp.SD)
    for c0, c1 in sp.cells():
        G = _geometry(sp, case, c0, c1)
        d = 0.0
        for a in range(3):
            for b in range(3):
                if G[a][b] is None:
                    continue
                v = G[a][b].expand(c1 - c0, sp.N, sp.N, sp.N)
                for k in range(3):
                    v = _con((t[a == k] * t[b == k]).T, v, k)
                d = d + v
        out.index_add_(0, sp.map(c0, c1).reshape(-1), d.reshape(-1))
    return torch.where(sp.constrained, torch.ones((), dtype=torch.float64, device=out.device), out)


def _chebyshev64(sp, case, b):
    """The smoother from zero and then one step, with its eigenvalue estimate (at most ten Jacobi-CG steps from
    (i mod 11) minus its mean, the largest Ritz value scaled by 1.2, range 15)."""
    geo = {c0: _geometry(sp, case, c0, c1) for c0, c1 in sp.cells()}
    inv = 1.0 / _diagonal64(sp, case)
    A = lambda v: _vmult64(sp, case, v, geo)  # noqa: E731
    r = torch.arange(sp.m, device=b.device).remainder(11).to(torch.float64)
    r = r - r.mean()
    z = inv * r
    rho, p, al, alphas, diag, off, beta, eba = float(r @ z), z, 0.0, [], [], [], 0.0, 0.0
    for it in range(1, 11):
        if it > 1:
            p = z + beta * p
        v = A(p)
        prev, al = al, rho / float(p @ v)
        r = r - al * v
        z = inv * r
        old, rho = rho, float(r @ z)
        if it > 1:
            diag.append(1.0 / prev + eba)
            eba = beta / prev
            off.append(math.sqrt(beta) / prev)
        beta = rho / old
        if float(r.norm()) <= 1e-10:
            break
    k = len(diag)
    T = np.diag(diag) + np.diag(off[:k - 1], 1) + np.diag(off[:k - 1], -1)
    hi = 1.2 * float(np.linalg.eigvalsh(T)[-1])
    lo = hi / 15.0
    theta, delta = 0.5 * (hi + lo), 0.5 * (hi - lo)

    def iterate(x, first, count):
        prev, x = x, x + first
        rhok = delta / theta
        for _ in range(count):
            rn = 1.0 / (2.0 * theta / delta - rhok)
            x, prev = x + rn * rhok * (x - prev) + 2.0 * rn / delta * inv * (b - A(x)), x
            rhok = rn
        return x

    x = iterate(torch.zeros_like(b), inv * b / theta, case["cheb"] - 1)
    return iterate(x, inv * (b - A(x)) / theta, case["cheb"] - 1)


def _transfer64(case, fine_src, coarse_src):
    fine = _Space(case, case["degree"]).number()
    if case["coarse_degree"]:
        co = _Space(case, case["coarse_degree"]).number()
        P = _t(_lagrange(co.xl, fine.xl)[0])
        patches = [(c0, c1, co.map(c0, c1), fine.map(c0, c1)) for c0, c1 in fine.cells()]
    else:
        co = _Space(case, case["degree"], case["refine"] - 1).number()
        nodes = np.concatenate([0.5 * co.xl, 0.5 + 0.5 * co.xl[1:]])
        P = _t(_lagrange(co.xl, nodes)[0])
        L0, L1 = fine.p * fine.n[0] + 1, fine.p * fine.n[1] + 1
        a = torch.arange(2 * co.p + 1, device=fine.dof.device)
        patches = []
        for c0, c1 in co.cells():
            x, y, z = (co.xyz[c0:c1, d, None] * 2 * co.p + a for d in range(3))
            patches.append((c0, c1, co.map(c0, c1),
                            fine.dof[(z[:, :, None, None] * L1 + y[:, None, :, None]) * L0 + x[:, None, None, :]]))
    zero = torch.zeros((), dtype=torch.float64, device=fine_src.device)
    mult = torch.zeros_like(fine_src)
    for _, _, _, fi in patches:
        mult.index_add_(0, fi.reshape(-1), torch.ones(fi.numel(), dtype=torch.float64, device=fi.device))
    w = torch.where(fine.constrained, zero, 1.0 / mult)
    cs = torch.where(co.constrained, zero, coarse_src)
    down, up = torch.zeros_like(coarse_src), torch.zeros_like(fine_src)
    for _, _, ci, fi in patches:
        r = (w * fine_src)[fi]
        q = cs[ci]
        for d in range(3):
            r = _con(P.T, r, d)
            q = _con(P, q, d)
        down.index_add_(0, ci.reshape(-1), r.reshape(-1))
        up.index_add_(0, fi.reshape(-1), (w[fi] * q).reshape(-1))
    return torch.where(co.constrained, zero, down), up


def _dg64(case, src):
    sp = _Space(case, case["degree"])
    N = sp.N
    S, SD = sp.S, sp.SD
    M, K = (S * sp.W) @ S.T, (SD * sp.W) @ SD.T
    ends = _lagrange(sp.xl, np.array([0.0, 1.0]))[1]
    dphi = [_t(ends[:, 0]), _t(ends[:, 1])]
    h, n = sp.h, sp.n
    place = (sp.xyz[:, 2] * n[1] + sp.xyz[:, 1]) * n[0] + sp.xyz[:, 0]
    u = torch.empty(sp.C, N, N, N, dtype=torch.float64, device=src.device)
    u[place] = src.reshape(sp.C, N, N, N)
    vol = h[0] * h[1] * h[2]
    mm = lambda v, dirs: _con(M, v, dirs[0]) if len(dirs) == 1 else _con(M, _con(M, v, dirs[0]), dirs[1])  # noqa: E731
    out = torch.zeros_like(u)
    for d in range(3):
        out += vol / h[d] ** 2 * mm(_con(K, u, d), [a for a in range(3) if a != d])
    c_pen = _penalty(case["degree"])
    for d in range(3):
        t = [a for a in range(3) if a != d]
        ax = 3 - d
        area = h[t[0]] * h[t[1]]
        sigma = c_pen / h[d]
        um = mm(u, t) * area  # the tangential mass applied once
        val = [um.select(ax, 0), um.select(ax, N - 1)]
        der = [torch.tensordot(um, dphi[s], dims=([ax], [0])) / h[d] for s in range(2)]
        g = lambda v: v.reshape(n[2], n[1], n[0], N, N)  # noqa: E731
        val, der = [g(v) for v in val], [g(v) for v in der]
        o = out.reshape(n[2], n[1], n[0], N, N, N)
        axis = 2 - d

        def test(cells, side, tv, tn):
            """Add tv phi + tn d_n phi on face `side` of the cells selected along `axis`."""
            view = o.narrow(axis, cells[0], cells[1])
            view.select(3 + 2 - d, 0 if side == 0 else N - 1).add_(tv)
            shape = [1] * 6
            shape[3 + 2 - d] = N
            view.add_(tn.unsqueeze(3 + 2 - d) * dphi[side].reshape(shape) * ((1.0 if side else -1.0) / h[d]))

        m = n[d]
        if m > 1:
            lo_v, hi_v = val[1].narrow(axis, 0, m - 1), val[0].narrow(axis, 1, m - 1)
            lo_d, hi_d = der[1].narrow(axis, 0, m - 1), der[0].narrow(axis, 1, m - 1)
            jump, avg = lo_v - hi_v, 0.5 * (lo_d + hi_d)
            test((0, m - 1), 1, sigma * jump - avg, -0.5 * jump)
            test((1, m - 1), 0, -(sigma * jump - avg), 0.5 * jump)
        for side, at in ((0, 0), (1, m - 1)):
            v, dn = val[side].narrow(axis, at, 1), der[side].narrow(axis, at, 1) * (1.0 if side else -1.0)
            test((at, 1), side, 2 * sigma * v - dn, -v)
    return out.reshape(sp.C, N, N, N)[place].reshape(-1)


def _solve64(sp, case, seed):
    """The solution of the linear system by Jacobi-CG to a residual of 1e-14."""
    f = sp.S @ sp.W
    cell = sp.h[0] * sp.h[1] * sp.h[2] * f[:, None, None] * f[None, :, None] * f[None, None, :]
    b = torch.zeros(sp.m, dtype=torch.float64, device=sp.dof.device)
    for c0, c1 in sp.cells():
        b.index_add_(0, sp.map(c0, c1).reshape(-1), cell.expand(c1 - c0, -1, -1, -1).reshape(-1))
    b = torch.where(sp.constrained, torch.zeros_like(b), b) * (1.0 + 0.5 * _uniform(sp.m, seed, torch.float64))
    geo = {c0: _geometry(sp, case, c0, c1) for c0, c1 in sp.cells()}
    inv = 1.0 / _diagonal64(sp, case)
    x, r = torch.zeros_like(b), b.clone()
    z = inv * r
    p, rho, stop = z, float(r @ z), 1e-14 * float(b.norm())
    for _ in range(1500):
        v = _vmult64(sp, case, p, geo)
        al = rho / float(p @ v)
        x, r = x + al * p, r - al * v
        if float(r.norm()) <= stop:
            break
        z = inv * r
        rho, old = float(r @ z), rho
        p = z + rho / old * p
    return x


def exact(case, seed):
    kind = case["kind"]
    torch.cuda.set_device(DEV)
    if kind in ("vmult", "smooth"):
        sp = _Space(case, case["degree"]).number()
        src = _uniform(sp.m, seed, _dt(case)[1]).to(torch.float64)
        return _vmult64(sp, case, src) if kind == "vmult" else _chebyshev64(sp, case, src)
    if kind == "dg":
        n = _sizes(case, case["degree"])[0] * (case["degree"] + 1) ** 3
        return _dg64(case, _uniform(n, seed, _dt(case)[1]).to(torch.float64))
    if kind == "transfer":
        nf = _sizes(case, case["degree"])[1]
        nc = _sizes(case, case["coarse_degree"])[1] if case["coarse_degree"] else _sizes(case, case["degree"], case["refine"] - 1)[1]
        tdt = _dt(case)[1]
        return _transfer64(case, _uniform(nf, seed, tdt).to(torch.float64), _uniform(nc, seed + 1, tdt).to(torch.float64))
    if kind == "solve" and case["geometry"] != "kappa" and _sizes(case, case["degree"])[1] <= 300_000:
        return _solve64(_Space(case, case["degree"]).number(), case, seed)
    return None  # a V-cycle has no value of its own; the large solves take too long without multigrid
