"""What a user of this library has it do, as cases that can be timed and checked.

Each case is one pass through the public entry points of
parallel-computing_b200/iga_b200.py, with inputs made on the GPU from a seed:

  matmul   y = A x with a plan that is kept (the MATSHELL MatMult)
  kappa    a new coefficient at the quadrature points, then a MatMult
           (a nonlinear or time-dependent coefficient)
  pc       z = M^-1 r with the exact bilinear-FEM preconditioner (the PCSHELL
           apply inside a caller's own Krylov loop)
  poisson  load vector and solve on a new right-hand side
  solve    solve for a given right-hand side
  batch    many independent solves together
  adjoint  forward solve, adjoint solve and dJ/dkappa (one step of an inversion)

Patches are rectangles whose sides, and quarter annuli whose radii, follow
from the seed. exact() restates every case in 64 bits with torch and numpy
alone: Cox-de Boor bases, the mapping's analytic derivatives, and dense 1-D
eigen-decompositions (or, with kappa, a plain preconditioned CG).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "parallel-computing_b200"))
import iga_b200 as ib  # noqa: E402

F64 = torch.float64
PREC = {"f64": ib.FP64, "f32": ib.FP32, "mixed": ib.MIXED}


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest MatMult in use: the p=2, 64 x 64 problem a Krylov loop
        # calls a hundred times; launches and latency count
        dict(name="matmul_p2_64", kind="matmul", p=2, nex=64, ney=64, prec="f64", fly=False, annulus=False),
        # the large FP64 MatMult with precomputed geometry (4.2 M unknowns)
        dict(name="matmul_p3_2048", kind="matmul", p=3, nex=2048, ney=2048, prec="f64", fly=False, annulus=False),
        # the on-the-fly MatMult (what a caller short of memory uses), ragged sizes
        dict(name="matmul_fly_p3_1021x773", kind="matmul", p=3, nex=1021, ney=773, prec="f64", fly=True,
             annulus=False),
        # the FP32 operator of a mixed-precision loop on a curved NURBS patch
        dict(name="matmul_f32_annulus_p4_1024", kind="matmul", p=4, nex=1024, ney=1024, prec="f32", fly=False,
             annulus=True),
        # a new coefficient field on a mid-sized patch, then the MatMult
        dict(name="kappa_p3_512", kind="kappa", p=3, nex=512, ney=512, prec="f64", fly=False),
        # the exact FEM preconditioner on its own, FP64 and (odd sizes) FP32
        dict(name="pc_p3_1024", kind="pc", p=3, nex=1024, ney=1024, prec="f64"),
        dict(name="pc_f32_p2_333x517", kind="pc", p=2, nex=333, ney=517, prec="f32"),
        # the reference's own configuration end to end: its load, p=2, 64 x 64,
        # inner Jacobi-CG on the FEM matrix as the preconditioner
        dict(name="poisson_p2_64_reference_pc", kind="poisson", p=2, nex=64, ney=64, prec="f64", pc="cg",
             annulus=False),
        # curved patch, manufactured load, mixed-precision refinement
        dict(name="poisson_mixed_annulus_p4_512", kind="poisson", p=4, nex=512, ney=512, prec="mixed", pc="exact",
             annulus=True),
        # the largest single solve: FP32 sweeps with FP64 refinement
        dict(name="solve_mixed_p3_2048", kind="solve", p=3, nex=2048, ney=2048, prec="mixed"),
        # 256 uneven solves of degree 2 and 3, 32 to 256 elements a side
        dict(name="batch_mixed_256", kind="batch", count=256, prec="mixed", shapes=2),
        # one gradient step for the coefficient of a p=3, 512 x 512 problem
        dict(name="adjoint_p3_512", kind="adjoint", p=3, nex=512, ney=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: degrees 1 to 5, sides from 16 elements
    up to the largest listed ones, square or not, both precisions and paths."""
    kind = rng.choice(["matmul"] * 4 + ["kappa", "pc", "pc", "poisson", "solve", "batch", "adjoint"])
    p = rng.choice([1, 2, 2, 3, 3, 3, 4, 5])

    def sides(lo, hi):
        a = _log(rng, lo, hi)
        return a, (a if rng.random() < 0.25 else min(hi, max(lo, int(a * math.exp(rng.uniform(-0.7, 0.7))))))

    if kind == "matmul":
        annulus = p >= 2 and rng.random() < 0.3
        a, b = sides(16, 2048 if p <= 3 else 1024)
        return dict(kind=kind, p=p, nex=a, ney=b, prec=rng.choice(["f64", "f32"]), fly=rng.random() < 0.4,
                    annulus=annulus)
    if kind == "kappa":
        a, b = sides(16, 1024 if p <= 3 else 512)
        return dict(kind=kind, p=p, nex=a, ney=b, prec=rng.choice(["f64", "f32"]), fly=rng.random() < 0.3)
    if kind == "pc":
        a, b = sides(16, 2048)
        return dict(kind=kind, p=p, nex=a, ney=b, prec=rng.choice(["f64", "f32"]))
    p = rng.choice([2, 3])
    if kind == "poisson":
        if rng.random() < 0.4:
            a, b = sides(16, 128)
            return dict(kind=kind, p=p, nex=a, ney=b, prec="f64", pc="cg", annulus=False)
        a, b = sides(32, 512)
        return dict(kind=kind, p=p, nex=a, ney=b, prec=rng.choice(["f64", "mixed"]), pc="exact",
                    annulus=rng.random() < 0.5)
    if kind == "solve":
        a, b = sides(32, 1024)
        return dict(kind=kind, p=p, nex=a, ney=b, prec=rng.choice(["f64", "mixed"]))
    if kind == "batch":
        return dict(kind=kind, count=_log(rng, 4, 256), prec=rng.choice(["f64", "mixed"]),
                    shapes=rng.randrange(3, 1000))
    a, b = sides(32, 512)
    return dict(kind="adjoint", p=p, nex=a, ney=b)


# ------------------------------------------------------------------ inputs
def _patch(case, seed):
    """Shape parameters of the patch: (Lx, Ly) of a rectangle, (r_in, r_out) of an annulus."""
    r = np.random.RandomState(seed % (1 << 31))
    if case.get("annulus"):
        return 1.0 + 0.2 * r.rand(), 2.0 + 0.4 * r.rand()
    return 0.8 + 0.4 * r.rand(), 0.8 + 0.4 * r.rand()


def _mesh(case, seed):
    a, b = _patch(case, seed)
    if case.get("annulus"):
        return ib.quarter_annulus(case["p"], case["nex"], case["ney"], a, b)
    return ib.unit_square(case["p"], case["nex"], case["ney"], a, b)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _ring(m, n):
    mask = torch.zeros(n, m, dtype=torch.bool, device="cuda")
    mask[0], mask[-1], mask[:, 0], mask[:, -1] = True, True, True, True
    return mask.reshape(-1)


def _kappa(case, seed):
    """A smooth positive coefficient at the quadrature points (element-major, qx
    fastest): the exponential of a sum of random waves, about one in size."""
    nq, nex, ney = case["p"] + 1, case["nex"], case["ney"]
    t = torch.from_numpy(np.polynomial.legendre.leggauss(nq)[0] * 0.5 + 0.5).cuda()
    x = ((torch.arange(nex, device="cuda", dtype=F64)[:, None] + t) / nex).view(1, nex, 1, nq)
    y = ((torch.arange(ney, device="cuda", dtype=F64)[:, None] + t) / ney).view(ney, 1, nq, 1)
    r = np.random.RandomState((seed + 77) % (1 << 31))
    g = torch.zeros(ney, nex, nq, nq, dtype=F64, device="cuda")
    for _ in range(6):
        kx, ky = r.randint(1, 6, 2)
        g += 0.4 * r.randn() * torch.cos(math.pi * kx * x + 6.28 * r.rand()) * torch.cos(math.pi * ky * y + 6.28 * r.rand())
    return torch.exp(g).reshape(-1)


def _inputs(case, seed):
    """The tensors of a pass (on the GPU), without the plan."""
    kind, gen = case["kind"], _gen(seed)
    if kind == "batch":
        parts = []
        for p, nex, ney in ib.batch_problems(case["count"], seed=case["shapes"]):
            b = torch.randn(ney + p, nex + p, dtype=F64, device="cuda", generator=gen)
            b[0], b[-1], b[:, 0], b[:, -1] = 0.0, 0.0, 0.0, 0.0
            parts.append(b.reshape(-1))
        return {"b": torch.cat(parts)}
    m, n = case["nex"] + case["p"], case["ney"] + case["p"]
    if kind == "poisson":
        return {}
    if kind == "adjoint":
        ring = _ring(m, n)
        y, x = torch.meshgrid(torch.linspace(0, 1, n, dtype=F64, device="cuda"),
                              torch.linspace(0, 1, m, dtype=F64, device="cuda"), indexing="ij")
        # observations: a smooth state and noise; the load is f = 2 pi^2 sin sin
        obs = (torch.sin(math.pi * x) * torch.sin(math.pi * y)).reshape(-1)
        obs = 0.9 * obs + 0.01 * torch.randn(m * n, dtype=F64, device="cuda", generator=gen)
        obs[ring] = 0.0
        return {"kappa": _kappa(case, seed), "obs": obs, "ring": ring}
    x = torch.rand(m * n, dtype=F64, device="cuda", generator=gen) * 2 - 1
    if kind == "solve":
        x[_ring(m, n)] = 0.0
    if case["prec"] == "f32":
        x = x.to(torch.float32)
    out = {"x": x}
    if kind == "kappa":
        out["kappa"] = _kappa(case, seed)
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = dict(_inputs(case, seed), case=case)
    if kind == "batch":
        meshes = [ib.unit_square(p, a, b) for p, a, b in ib.batch_problems(case["count"], seed=case["shapes"])]
        s["batch"] = ib.Batch(meshes, precision=PREC[case["prec"]], tune_file=ib.TUNE_FILE)
        s["y"] = torch.empty_like(s["b"])
        return s
    mesh = _mesh(case, seed)
    prec = ib.FP64 if kind == "adjoint" else PREC[case["prec"]]
    if kind == "pc":
        prec = ib.FP64   # the preconditioner's precision is an argument of the call
    s["plan"] = ib.Plan(mesh, precision=prec, geometry=ib.GEOM_ON_THE_FLY if case.get("fly") else ib.GEOM_PRECOMPUTED)
    if kind == "poisson":
        s["b"] = torch.empty(s["plan"].nfunc, dtype=F64, device="cuda")
        s["y"] = torch.empty_like(s["b"])
    elif kind == "adjoint":
        s["F"] = torch.empty(s["plan"].nfunc, dtype=F64, device="cuda")
        s["plan"].rhs(s["F"], ib.F_SINSIN)
        s["step"] = ib.kappa_solve_function()
    else:
        s["y"] = torch.empty_like(s["x"])
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "matmul":
        s["plan"].apply(s["x"], s["y"])
        return s["y"]
    if kind == "kappa":
        s["plan"].set_kappa(s["kappa"])
        s["plan"].apply(s["x"], s["y"])
        return s["y"]
    if kind == "pc":
        s["plan"].pc_apply(s["x"], s["y"], pc=ib.PC_FEM_EXACT, precision=PREC[case["prec"]])
        return s["y"]
    if kind == "poisson":
        s["plan"].rhs(s["b"], ib.F_ANNULUS if case["annulus"] else ib.F_REFERENCE)
        s["plan"].solve(s["b"], s["y"], precision=PREC[case["prec"]],
                        pc=ib.PC_FEM_CG if case["pc"] == "cg" else ib.PC_FEM_EXACT)
        return {"load": s["b"], "u": s["y"]}
    if kind == "solve":
        s["plan"].solve(s["x"], s["y"], precision=PREC[case["prec"]], pc=ib.PC_FEM_EXACT)
        return s["y"]
    if kind == "batch":
        s["batch"].solve(s["b"], s["y"], precision=PREC[case["prec"]])
        return s["y"]
    kappa = s["kappa"].clone().requires_grad_(True)
    u = s["step"].apply(kappa, s["plan"], s["F"], s["ring"], dict(pc=ib.PC_FEM_EXACT, rtol=1e-10))
    J = 0.5 * ((u - s["obs"]) ** 2).sum()
    J.backward()
    return {"u": u.detach(), "grad": kappa.grad}


def work(case):
    """Bytes: vectors and (where the plan or the call has them) geometry or
    coefficients once. Flops: one sum-factorised operator pass, the exact FEM
    inverse's two transforms, or one of each for a solve."""
    def apply_flops(p, ne):
        nb = p + 1   # two 1-D contractions in, the 2x2 factor, two out
        return ne * (8.0 * nb * nb + 8.0 * nb * nb * nb + 6.0 * nb * nb)

    if case["kind"] == "batch":
        shapes = ib.batch_problems(case["count"], seed=case["shapes"])
        dof = sum((a + p) * (b + p) for p, a, b in shapes)
        geo = sum(3 * 8 * (p + 1) ** 2 * a * b for p, a, b in shapes)
        fl = sum(apply_flops(p, a * b) + 4.0 * (a + p) ** 2 * (b + p) for p, a, b in shapes)
        return {"bytes": 16.0 * dof + geo, "flops": fl}
    p, nex, ney = case["p"], case["nex"], case["ney"]
    es = 4 if case.get("prec") == "f32" else 8
    m, n, ne, nq2 = nex + p, ney + p, nex * ney, (p + 1) ** 2
    if case["kind"] == "matmul":
        geo = 2 * es * m * n if case["fly"] else 3 * es * nq2 * ne
        return {"bytes": 2.0 * es * m * n + geo, "flops": apply_flops(p, ne) * (2 if case["fly"] else 1)}
    if case["kind"] == "kappa":   # kappa in, x in, y out
        return {"bytes": 8.0 * nq2 * ne + 2.0 * es * m * n, "flops": 2 * apply_flops(p, ne)}
    pc = 4.0 * (m - 2) ** 2 * (n - 2)   # two transforms of n vectors of length m
    if case["kind"] == "pc":   # half the flops: the x eigenvectors are even or odd
        return {"bytes": 2.0 * es * m * n + es * m * m / 2, "flops": pc / 2}
    if case["kind"] == "adjoint":
        return {"bytes": 2 * 8.0 * nq2 * ne + 3 * 8.0 * m * n, "flops": 3 * apply_flops(p, ne) + pc}
    return {"bytes": 16.0 * m * n + 24.0 * nq2 * ne, "flops": apply_flops(p, ne) + pc / 2}


# ------------------------------------------------------------------ 64-bit restatement
def _gauss(nq):
    t, w = np.polynomial.legendre.leggauss(nq)
    return 0.5 * t + 0.5, 0.5 * w


def _knots(p, ne):
    return np.concatenate([np.zeros(p), np.linspace(0.0, 1.0, ne + 1), np.ones(p)])


def _basis(p, ne, at=None):
    """Values and element-local derivatives [ne, points, p + 1] of the open
    uniform B-splines of degree p at the points `at` of every element."""
    at = _gauss(p + 1)[0] if at is None else at
    U = _knots(p, ne)
    x = (np.arange(ne)[:, None] + at[None, :]) / ne          # [ne, nq]
    e = np.arange(ne)[:, None]
    N = [np.ones_like(x)]
    low = None
    for d in range(1, p + 1):
        if d == p:
            low = N
        new = [np.zeros_like(x) for _ in range(d + 1)]
        for k in range(d):        # N[k] is the degree d-1 function of index e + p - (d-1) + k
            i = e + p - d + 1 + k
            left, right = U[i], U[i + d]
            a = N[k] / (right - left)
            new[k] = new[k] + (right - x) * a
            new[k + 1] = new[k + 1] + (x - left) * a
        N = new
    D = [np.zeros_like(x) for _ in range(p + 1)]
    for k in range(p):
        i = e + 1 + k
        a = p * low[k] / (U[i + p] - U[i])
        D[k] = D[k] - a
        D[k + 1] = D[k + 1] + a
    return np.stack(N, -1), np.stack(D, -1) / ne


def _directions(case, seed):
    """Per direction: value and derivative tables, and the 1-D factors g0 (times
    derivative x derivative) and g1 (times value x value) of the separable
    G = w det(J) J^-1 J^-T; and x(q), y(q), det(q) for the load."""
    p, nex, ney = case["p"], case["nex"], case["ney"]
    a, b = _patch(case, seed)
    t, w = _gauss(p + 1)
    vx, dx = _basis(p, nex)
    vy, dy = _basis(p, ney)
    xi = (np.arange(nex)[:, None] + t) / nex
    eta = (np.arange(ney)[:, None] + t) / ney
    if not case.get("annulus"):
        one_x, one_y = np.ones_like(xi), np.ones_like(eta)
        hx, hy = a / nex, b / ney
        # G00 = w hy/hx, G11 = w hx/hy
        return (vx, dx, one_x / hx * w, one_x * hx * w), (vy, dy, one_y / hy * w, one_y * hy * w), \
            (a * xi, b * eta, one_x * hx * w, one_y * hy * w)
    # x = r(xi) (cos, sin)(theta(eta)), rational quadratic arc with middle weight sqrt(1/2)
    s2 = math.sqrt(0.5)

    def wfun(z):
        return (1 - z) ** 2 + 2 * s2 * z * (1 - z) + z ** 2

    # weights of the refined basis: the spline that equals wfun, by interpolation
    grev = np.array([_knots(p, ney)[i + 1:i + p + 1].mean() for i in range(ney + p)])
    A = np.zeros((ney + p, ney + p))
    cell = np.minimum((grev * ney).astype(int), ney - 1)
    for i, (g, c) in enumerate(zip(grev, cell)):
        A[i, c:c + p + 1] = _basis_at(p, ney, c, g)
    wt = np.linalg.solve(A, wfun(grev))
    wloc = np.stack([wt[k:k + ney] for k in range(p + 1)], -1)[:, None, :]
    W, dW = (vy * wloc).sum(-1, keepdims=True), (dy * wloc).sum(-1, keepdims=True)
    ry = vy * wloc / W
    rdy = (dy * wloc - dW * ry) / W
    c, s = (1 - eta) ** 2 + 2 * s2 * eta * (1 - eta), eta ** 2 + 2 * s2 * eta * (1 - eta)
    # theta' = (c s' - c' s) / (c^2 + s^2), per element
    dc, ds = -2 * (1 - eta) + 2 * s2 * (1 - 2 * eta), 2 * eta + 2 * s2 * (1 - 2 * eta)
    dth = (c * ds - dc * s) / (c * c + s * s) / ney
    r, dr = a + (b - a) * xi, (b - a) / nex
    th = np.arctan2(s, c)
    # det = r r' theta', G00 = w r theta' / r', G11 = w r' / (r theta')
    return (vx, dx, r / dr * w, dr / r * w), (ry, rdy, w / dth, dth * w), (r, th, r * dr * w, dth * w)


def _basis_at(p, ne, cell, x):
    v, _ = _basis(p, ne, np.array([x * ne - cell]))
    return v[cell, 0]


def _cuda(*arrays):
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in arrays]


def _separable_G(X, Y):
    """(g00x, g11x, g00y, g11y): G00(q) = g00x[x] g00y[y] and G11(q) = g11x[x] g11y[y].
    G00 pairs x's derivative factor with y's value factor, G11 the other way round."""
    return _cuda(X[2], X[3], Y[3], Y[2])


def _apply(case, X, Y, x, kappa=None):
    """K x (SPD sign, no boundary rule), matrix-free in slabs of element rows."""
    p, nex, ney = case["p"], case["nex"], case["ney"]
    nb, m, n = p + 1, nex + p, ney + p
    vx, dx = _cuda(X[0], X[1])
    vy, dy = _cuda(Y[0], Y[1])
    g00x, g11x, g00y, g11y = _separable_G(X, Y)
    x = x.reshape(n, m)
    y = torch.zeros(n, m, dtype=F64, device="cuda")
    rows = max(1, (1 << 21) // nex)
    for e0 in range(0, ney, rows):
        e1 = min(ney, e0 + rows)
        U = x[e0:e1 + p].unfold(0, nb, 1).unfold(1, nb, 1)          # [ey, ex, j, i]
        ux = torch.einsum("yxji,xai->yxja", U, dx)
        uv = torch.einsum("yxji,xai->yxja", U, vx)
        gx = torch.einsum("yxja,ybj->yxba", ux, vy[e0:e1])
        gy = torch.einsum("yxja,ybj->yxba", uv, dy[e0:e1])
        gx = gx * (g00x[None, :, None, :] * g00y[e0:e1, None, :, None])
        gy = gy * (g11x[None, :, None, :] * g11y[e0:e1, None, :, None])
        if kappa is not None:
            k = kappa.reshape(ney, nex, nb, nb)[e0:e1]
            gx, gy = gx * k, gy * k
        out = torch.einsum("yxja,xai->yxji", torch.einsum("yxba,ybj->yxja", gx, vy[e0:e1]), dx)
        out += torch.einsum("yxja,xai->yxji", torch.einsum("yxba,ybj->yxja", gy, dy[e0:e1]), vx)
        for j in range(nb):
            for i in range(nb):
                y[e0 + j:e1 + j, i:i + nex] += out[:, :, j, i]
    return y.reshape(-1)


def _grad_product(case, X, Y, u, lam):
    """-(grad lam . grad u) JxW at the quadrature points."""
    p, nex, ney = case["p"], case["nex"], case["ney"]
    nb, m, n = p + 1, nex + p, ney + p
    vx, dx = _cuda(X[0], X[1])
    vy, dy = _cuda(Y[0], Y[1])
    g00x, g11x, g00y, g11y = _separable_G(X, Y)

    def grads(v):
        U = v.reshape(n, m).unfold(0, nb, 1).unfold(1, nb, 1)
        return (torch.einsum("yxja,ybj->yxba", torch.einsum("yxji,xai->yxja", U, dx), vy),
                torch.einsum("yxja,ybj->yxba", torch.einsum("yxji,xai->yxja", U, vx), dy))

    (ux, uy), (lx, ly) = grads(u), grads(lam)
    g = ux * lx * (g00x[None, :, None, :] * g00y[:, None, :, None])
    g += uy * ly * (g11x[None, :, None, :] * g11y[:, None, :, None])
    return -g.reshape(-1)


def _assemble_1d(T, f, ne):
    """sum_q f(e, q) T_i T_j as a dense matrix."""
    T, f = _cuda(T, f)
    nb = T.shape[-1]
    L = torch.einsum("eqi,eqj,eq->eij", T, T, f)
    A = torch.zeros(ne + nb - 1, ne + nb - 1, dtype=F64, device="cuda")
    e = torch.arange(ne, device="cuda")
    for i in range(nb):
        for j in range(nb):
            A[e + i, e + j] += L[:, i, j]
    return A


class _FastDiagonal:
    """(Kx (x) My + Mx (x) Ky)^-1 on the interior by dense generalised eigenpairs of each direction."""

    def __init__(self, Kx, Mx, Ky, My):
        self.lx, self.Vx = self._pairs(Kx, Mx)
        self.ly, self.Vy = self._pairs(Ky, My)

    @staticmethod
    def _pairs(K, M):
        L = torch.linalg.cholesky(M)
        A = torch.linalg.solve_triangular(L, K, upper=False)
        A = torch.linalg.solve_triangular(L, A.T.contiguous(), upper=False)
        lam, Q = torch.linalg.eigh(0.5 * (A + A.T))
        return lam, torch.linalg.solve_triangular(L.T.contiguous(), Q, upper=True)

    def __call__(self, b):   # b: [ny, nx]
        T = self.Vy.T @ b @ self.Vx
        return self.Vy @ (T / (self.ly[:, None] + self.lx[None, :])) @ self.Vx.T


def _solver(case, X, Y):
    """u = K^-1 b on the free control points (boundary values of b kept), kappa = 1."""
    nex, ney = case["nex"], case["ney"]

    def inner(A):
        return A[1:-1, 1:-1].contiguous()

    # K = (x: g00, der der) (y: g00 of y, val val) + (x: g11, val val) (y: der der)
    fd = _FastDiagonal(inner(_assemble_1d(X[1], X[2], nex)), inner(_assemble_1d(X[0], X[3], nex)),
                       inner(_assemble_1d(Y[1], Y[2], ney)), inner(_assemble_1d(Y[0], Y[3], ney)))
    m, n = nex + case["p"], ney + case["p"]

    def solve(b):
        z = b.reshape(n, m).clone()
        z[1:-1, 1:-1] = fd(z[1:-1, 1:-1])
        return z.reshape(-1)
    return solve


def _fem_nodes(p, ne, L):
    """Nodes of the bilinear FEM grid: Greville abscissae of degree p - 2 on ne + 2 uniform spans (p >= 3), else of degree p."""
    d, spans = (p - 2, ne + 2) if p >= 3 else (p, ne)
    U = _knots(d, spans)
    return L * np.array([U[i + 1:i + d + 1].mean() for i in range(spans + d)])


def _fem_1d(g):
    h = np.diff(g)
    n = len(g)
    K, M = np.zeros((n, n)), np.zeros((n, n))
    for e in range(n - 1):
        K[e:e + 2, e:e + 2] += np.array([[1, -1], [-1, 1]]) / h[e]
        M[e:e + 2, e:e + 2] += np.array([[2, 1], [1, 2]]) * h[e] / 6
    return _cuda(K[1:-1, 1:-1], M[1:-1, 1:-1])


def _load(case, X, Y, geo, annulus):
    """F = int R f, zero on the boundary ring."""
    p, nex, ney = case["p"], case["nex"], case["ney"]
    nb, m, n = p + 1, nex + p, ney + p
    a, b, wx, wy = _cuda(*geo)
    vx, vy = _cuda(X[0], Y[0])
    out = torch.zeros(n, m, dtype=F64, device="cuda")
    rows = max(1, (1 << 21) // nex)
    A = a[None, :, None, :]
    for e0 in range(0, ney, rows):
        e1 = min(ney, e0 + rows)
        B = b[e0:e1, None, :, None]
        if annulus:   # A = r, B = theta
            pr = math.pi * A
            f = (math.pi ** 2 * torch.sin(pr) - math.pi * torch.cos(pr) / A + 4 * torch.sin(pr) / A ** 2) * torch.sin(2 * B)
        else:
            f = A * (1 - A) * B * (1 - B)
        f = f * (wx[None, :, None, :] * wy[e0:e1, None, :, None])
        L = torch.einsum("yxba,xai,ybj->yxji", f, vx, vy[e0:e1])
        for j in range(nb):
            for i in range(nb):
                out[e0 + j:e1 + j, i:i + nex] += L[:, :, j, i]
    out = out.reshape(-1)
    out[_ring(m, n)] = 0.0
    return out


def _pcg(A, M, b, tol, most):
    x = torch.zeros_like(b)
    r = b.clone()
    z = M(r)
    p = z.clone()
    rz = torch.dot(r, z)
    stop = float(rz) * tol * tol
    for _ in range(most):
        q = A(p)
        al = rz / torch.dot(p, q)
        x += al * p
        r -= al * q
        z = M(r)
        new = torch.dot(r, z)
        if float(new) <= stop:
            break
        p = z + (new / rz) * p
        rz = new
    return x


def exact(case, seed):
    kind = case["kind"]
    s = _inputs(case, seed)
    if kind == "batch":
        parts, at, pairs = [], 0, {}
        for p, nex, ney in ib.batch_problems(case["count"], seed=case["shapes"]):
            def one_d(ne):
                if (p, ne) not in pairs:
                    v, d = _basis(p, ne)
                    f = np.ones((ne, 1)) * _gauss(p + 1)[1]
                    pairs[p, ne] = _FastDiagonal._pairs(_assemble_1d(d, f * ne, ne)[1:-1, 1:-1].contiguous(),
                                                        _assemble_1d(v, f / ne, ne)[1:-1, 1:-1].contiguous())
                return pairs[p, ne]
            fd = _FastDiagonal.__new__(_FastDiagonal)
            (fd.lx, fd.Vx), (fd.ly, fd.Vy) = one_d(nex), one_d(ney)
            m, n = nex + p, ney + p
            z = s["b"][at:at + m * n].reshape(n, m).clone()
            z[1:-1, 1:-1] = fd(z[1:-1, 1:-1])
            parts.append(z.reshape(-1))
            at += m * n
        return torch.cat(parts)
    m, n = case["nex"] + case["p"], case["ney"] + case["p"]
    if kind == "pc":
        a, b = _patch(case, seed)
        fd = _FastDiagonal(*_fem_1d(_fem_nodes(case["p"], case["nex"], a)),
                           *_fem_1d(_fem_nodes(case["p"], case["ney"], b)))
        z = s["x"].double().reshape(n, m).clone()
        z[1:-1, 1:-1] = fd(z[1:-1, 1:-1])
        return z.reshape(-1)
    X, Y, geo = _directions(case, seed)
    ring = _ring(m, n)
    if kind in ("matmul", "kappa"):
        y = -_apply(case, X, Y, s["x"].double(), s.get("kappa"))
        y[ring] = 0.0
        return y
    if kind == "poisson":
        F = _load(case, X, Y, geo, case["annulus"])
        return {"load": F, "u": _solver(case, X, Y)(F)}
    solve = _solver(case, X, Y)
    if kind == "solve":
        return solve(s["x"])
    # adjoint: the same solves by CG with the kappa = 1 inverse as preconditioner
    xq, yq, wx, wy = geo
    f = 2 * math.pi ** 2 * np.sin(math.pi * yq)[:, None, :, None] * np.sin(math.pi * xq)[None, :, None, :]
    f, vx, vy = _cuda(f * wy[:, None, :, None] * wx[None, :, None, :], X[0], Y[0])
    L = torch.einsum("yxba,xai,ybj->yxji", f, vx, vy)
    F = torch.zeros(n, m, dtype=F64, device="cuda")
    for j in range(case["p"] + 1):
        for i in range(case["p"] + 1):
            F[j:j + case["ney"], i:i + case["nex"]] += L[:, :, j, i]
    F = F.reshape(-1)
    F[ring] = 0.0

    def A(v):
        y = _apply(case, X, Y, torch.where(ring, torch.zeros_like(v), v), s["kappa"])
        return torch.where(ring, v, y)

    u = _pcg(A, solve, F, 1e-13, 400)
    rhs = u - s["obs"]
    rhs[ring] = 0.0
    lam = _pcg(A, solve, rhs, 1e-13, 400)
    return {"u": u, "grad": _grad_product(case, X, Y, u, lam)}
