"""The kernels' and launch rules' edges: sizes where a rule on the patch's size
switches, remainders of tiles and the smallest patches, each against the oracle.

Bars: FP64 1e-12 and FP32 2e-5 relative to the largest entry, as everywhere
for the MatMult.
"""
import numpy as np
import pytest

from iga_testlib import distorted, load_binding, splitmix_uniform

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch_cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.fixture(scope="module")
def ib():
    return load_binding()


def rel(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


# The strip height of patches of up to one wave of strips: one element, fewer
# rows than the shortest strip, 2-row strips, ragged last strips, the last
# square p = 3 patch the rule takes (42 columns of 42 strips on 148 SMs of 12
# warps) and the first one past it.
@pytest.mark.parametrize("p,nex,ney", [(1, 1, 1), (1, 64, 65), (2, 3, 1), (2, 257, 9), (3, 17, 2), (3, 31, 128),
                                       (4, 40, 23), (5, 33, 6), (3, 672, 672), (3, 688, 688)])
@pytest.mark.parametrize("geom", [0, 1])
def test_strip_height_of_small_patches(torch_cuda, ib, orc, p, nex, ney, geom):
    M = distorted(ib.unit_square(p, nex, ney))
    x = splitmix_uniform(p * 100 + nex, -1.0, 1.0, (nex + p) * (ney + p))
    ref = orc.apply_mf(M, x)
    plan = ib.Plan(M, precision=ib.MIXED, geometry=geom)
    # FP32 on-the-fly geometry differences FP32 control points over one element:
    # its error grows with the element count, so FP32 is held to its bar with
    # precomputed geometry (same strips, same kernel body)
    bars = [(ib.FP64, torch_cuda.float64, 1e-12), (ib.FP32, torch_cuda.float32, 2e-5)]
    for prec, dt, tol in bars if geom == ib.GEOM_PRECOMPUTED else bars[:1]:
        xd = torch_cuda.from_numpy(x).to("cuda", dt)
        yd = torch_cuda.full_like(xd, float("nan"))
        plan.apply(xd, yd, precision=prec)
        assert rel(yd.double().cpu().numpy(), ref) < tol
    plan.close()


# The inner FEM-CG in one cluster: one row per thread (40 x 1), two (1 x 1),
# four (64^2) and eight (300 x 125), fewer grid rows than CTAs, a 3-node direction, the first sizes past
# the cluster (600 x 300: the launch-per-step path). Its stop is the recurrence
# residual at pc_rtol; the true residual may exceed it by the rounding of the
# iteration, well under pc_rtol itself in FP64 (condition ~ 1e4 x 1e-16); in
# FP32 (condition 4e3 x 6e-8 = 2.4e-4) under a pc_rtol of 1e-3.
@pytest.mark.parametrize("p,nex,ney", [(2, 64, 64), (2, 1, 1), (3, 40, 1), (1, 2, 30), (2, 17, 90), (3, 96, 128),
                                       (2, 255, 62), (3, 300, 125), (2, 600, 300)])
@pytest.mark.parametrize("prec", [0, 1])
def test_fem_cg_in_a_cluster(torch_cuda, ib, orc, p, nex, ney, prec):
    plan = ib.Plan(ib.unit_square(p, nex, ney))
    gx, gy = plan.fem_nodes()
    r = splitmix_uniform(p + 7 * nex, -1.0, 1.0, plan.nfunc)   # boundary entries not zero
    dt = torch_cuda.float32 if prec else torch_cuda.float64
    rd = torch_cuda.from_numpy(r).to("cuda", dt)
    zd = torch_cuda.full_like(rd, float("nan"))
    tol = 1e-3 if prec else 1e-10
    plan.pc_apply(rd, zd, pc=ib.PC_FEM_CG, precision=prec, pc_rtol=tol)
    rr = rd.double().cpu().numpy()
    res = orc.fem_matvec(gx, gy, zd.double().cpu().numpy()) - rr
    assert np.linalg.norm(res) <= 2 * tol * np.linalg.norm(rr)
    # the same call twice gives the same bits
    z2 = torch_cuda.full_like(rd, float("nan"))
    plan.pc_apply(rd, z2, pc=ib.PC_FEM_CG, precision=prec, pc_rtol=tol)
    assert torch_cuda.equal(zd, z2)
    plan.close()


def test_fem_cg_breakdown_and_zero(torch_cuda, ib):
    plan = ib.Plan(ib.unit_square(2, 40, 33))
    r = torch_cuda.ones(plan.nfunc, dtype=torch_cuda.float64, device="cuda")
    r[500] = float("nan")
    z = torch_cuda.full_like(r, 3.0)
    with pytest.raises(ib.IgaError):
        plan.pc_apply(r, z, pc=ib.PC_FEM_CG)
    assert torch_cuda.equal(z, torch_cuda.full_like(r, 3.0))   # left as it was
    r.zero_()
    plan.pc_apply(r, z, pc=ib.PC_FEM_CG)
    assert float(z.abs().max()) == 0.0
    plan.close()


# Quadrature-point fields: one element, fewer columns or rows than a strip or
# a chunk, remainders of 16 columns, 8 rows, 32 x 8 and 32-column tiles, every
# degree (its own kernel and G layout), both precisions' G on strips of
# their own heights.
FIELD_SHAPES = [(1, 1, 1), (1, 33, 40), (2, 16, 8), (2, 50, 37), (3, 15, 9), (3, 64, 65), (4, 17, 31), (4, 70, 20),
                (5, 33, 18), (5, 7, 90)]


@pytest.mark.parametrize("p,nex,ney", FIELD_SHAPES)
def test_set_kappa_adjoint_gradient_and_load(torch_cuda, ib, orc, p, nex, ney):
    M = distorted(ib.unit_square(p, nex, ney))
    plan = ib.Plan(M, precision=ib.MIXED)
    n = plan.nfunc
    kq = np.exp(splitmix_uniform(5, -1.0, 1.0, nex * ney * (p + 1) ** 2))
    x = splitmix_uniform(6, -1.0, 1.0, n)
    lam = splitmix_uniform(7, -1.0, 1.0, n)
    plan.set_kappa(torch_cuda.from_numpy(kq).cuda())
    ref = orc.apply_mf(dict(M, kappa=kq), x)
    for prec, dt, tol in ((ib.FP64, torch_cuda.float64, 1e-12), (ib.FP32, torch_cuda.float32, 2e-5)):
        xd = torch_cuda.from_numpy(x).to("cuda", dt)
        yd = torch_cuda.full_like(xd, float("nan"))
        plan.apply(xd, yd, precision=prec)
        assert rel(yd.double().cpu().numpy(), ref) < tol
    g = torch_cuda.full((kq.size,), float("nan"), dtype=torch_cuda.float64, device="cuda")
    plan.adjoint_grad(torch_cuda.from_numpy(x).cuda(), torch_cuda.from_numpy(lam).cuda(), g)
    assert rel(g.cpu().numpy(), orc.adjoint_grad(M, x, lam)) < 1e-12
    F = torch_cuda.full((n,), float("nan"), dtype=torch_cuda.float64, device="cuda")
    for kind in (ib.F_REFERENCE, ib.F_SINSIN):
        plan.rhs(F, kind)
        assert np.abs(F.cpu().numpy() - orc.rhs(M, kind)).max() <= 1e-12 * max(np.abs(orc.rhs(M, kind)).max(), 1e-300)
    plan.close()


# Seams: a strip height that leaves one row (or fewer than P) in the last
# strip row, one strip row or column only, more than one block of points per
# seam in either direction.
@pytest.mark.parametrize("p,nex,ney,ty", [(3, 33, 9, 4), (3, 17, 5, 4), (2, 16, 30, 7), (4, 40, 4, 5), (5, 49, 11, 5),
                                          (1, 600, 3, 2), (3, 32, 200, 199), (2, 130, 300, 16)])
@pytest.mark.parametrize("bc", [0, 1, 2])
def test_seams(torch_cuda, ib, orc, p, nex, ney, ty, bc):
    M = distorted(ib.unit_square(p, nex, ney))
    plan = ib.Plan(M, bc=bc, sign=1, rows_per_strip=ty)
    x = splitmix_uniform(p + nex, -1.0, 1.0, plan.nfunc)
    xd = torch_cuda.from_numpy(x).cuda()
    yd = torch_cuda.full_like(xd, float("nan"))
    plan.apply(xd, yd)
    ref = orc.apply_mf(M, x, sign=1.0, bc=0 if bc == 2 else bc)
    y, m, n = yd.cpu().numpy(), nex + p, ney + p
    if bc == 2:   # full sums on the ring too: compare the interior, the ring with tall strips
        one = ib.Plan(M, bc=bc, sign=1, rows_per_strip=max(ney, p))
        y2 = torch_cuda.full_like(xd, float("nan"))
        one.apply(xd, y2)
        assert rel(y, y2.cpu().numpy()) < 1e-12
        inner = np.s_[1:-1, 1:-1]
        y, ref = y.reshape(n, m)[inner], ref.reshape(n, m)[inner]
    assert rel(y, ref) < 1e-12
    # a caller's own capture, replayed
    g = torch_cuda.cuda.CUDAGraph()
    s = torch_cuda.cuda.Stream()
    y3 = torch_cuda.full_like(xd, float("nan"))
    with torch_cuda.cuda.graph(g, stream=s):
        plan.apply(xd, y3, stream=s)
    g.replay()
    torch_cuda.cuda.synchronize()
    assert torch_cuda.equal(y3, yd)


# The exact preconditioner's FP64 GEMM tiles: 32 x 32 (small and ragged sizes,
# 700^2) and 64 x 64 (1022^2, whose half transforms give every SM two), one
# tile and less, with and without the parity split; and the solver's loop on
# it with and without a kappa scaling (r.z taken in the unfold or not).
# K_fem z = r to 1e-10 as for every exact inverse.
@pytest.mark.parametrize("p,nex,ney", [(2, 5, 9), (2, 31, 33), (3, 65, 200), (3, 700, 690), (3, 1021, 1021)])
@pytest.mark.parametrize("split", [0, 1])
def test_exact_preconditioner_tiles(torch_cuda, ib, orc, p, nex, ney, split):
    plan = ib.Plan(ib.unit_square(p, nex, ney))
    plan.set_pc_split(split)
    gx, gy = plan.fem_nodes()
    r = splitmix_uniform(p + nex, -1.0, 1.0, plan.nfunc)
    rd = torch_cuda.from_numpy(r).cuda()
    zd = torch_cuda.full_like(rd, float("nan"))
    plan.pc_apply(rd, zd)
    res = orc.fem_matvec(gx, gy, zd.cpu().numpy()) - r
    assert np.linalg.norm(res) <= 1e-10 * np.linalg.norm(r)
    if nex > 300:
        plan.close()
        return
    # z = S M^-1 S r with S from kappa, through the same kernels (kappa = 4: S = 1/2)
    kq = torch_cuda.full((nex * ney * (p + 1) ** 2,), 4.0, dtype=torch_cuda.float64, device="cuda")
    plan.set_kappa(kq)
    z2 = torch_cuda.full_like(rd, float("nan"))
    plan.pc_apply(rd, z2)
    assert rel(z2.cpu().numpy(), 0.25 * zd.cpu().numpy()) < 1e-12
    plan.close()
    plan = ib.Plan(ib.unit_square(p, nex, ney), precision=ib.MIXED)
    plan.set_pc_split(split)
    m, n = nex + p, ney + p
    b = r.reshape(n, m).copy()
    b[0], b[-1], b[:, 0], b[:, -1] = 0.0, 0.0, 0.0, 0.0
    bd = torch_cuda.from_numpy(b.ravel()).cuda()
    ref = None
    for kappa in (False, True):
        if kappa:
            plan.set_kappa(kq)
        for prec in (ib.FP64, ib.MIXED, ib.MIXED_PC):
            x = torch_cuda.zeros_like(bd)
            st = plan.solve(bd, x, precision=prec, pc=ib.PC_FEM_EXACT)
            assert st.relres <= 1e-10
            x = x.cpu().numpy() * (4.0 if kappa else 1.0)
            ref = x if ref is None else ref
            # K's condition times the residuals' 1e-10 bounds the difference; 1e-7 holds it with room
            assert rel(x, ref) < 1e-7
    plan.close()


# The batched exact preconditioner at the edges of its row segments (one row,
# segments without rows, full ones, 272 rows), of its 32-mode blocks and of
# its GEMM tiles and k slices (31 to 33, 64, 65, 128, 129 and 257 modes).
# FP64: K_fem z = r to 1e-10; FP32, on TF32 operands, 1e-2 of the FP64 z.
def test_batch_preconditioner_edges(torch_cuda, ib, orc):
    free = [(1, 1), (31, 16), (32, 17), (33, 33), (64, 145), (65, 15), (128, 271), (129, 272), (257, 63), (2, 129)]
    meshes = [ib.unit_square(p, nx + 2 - p, ny + 2 - p) for i, (nx, ny) in enumerate(free) for p in [1 if min(nx, ny) < 2 else 1 + i % 2]]
    batch = ib.Batch(meshes, precision=ib.MIXED)
    r = splitmix_uniform(29, -1.0, 1.0, batch.ntot)
    rd = torch_cuda.from_numpy(r).cuda()
    zd = torch_cuda.full_like(rd, float("nan"))
    batch.pc_apply(rd, zd)
    z32 = torch_cuda.full_like(rd.float(), float("nan"))
    batch.pc_apply(rd.float(), z32, precision=ib.FP32)
    z, z32 = zd.cpu().numpy(), z32.double().cpu().numpy()
    for i, m in enumerate(meshes):
        a, b = batch.offsets[i], batch.offsets[i + 1]
        plan = ib.Plan(m)
        gx, gy = plan.fem_nodes()
        plan.close()
        res = orc.fem_matvec(gx, gy, z[a:b]) - r[a:b]
        assert np.linalg.norm(res) <= 1e-10 * np.linalg.norm(r[a:b]), free[i]
        assert rel(z32[a:b], z[a:b]) < 1e-2, free[i]
    batch.close()


# The batched iteration's vector kernels: patches that start at every entry
# offset of a 16-byte word, shorter than a word's ragged ends, of exactly one
# chunk of 2048 entries (32 x 64 control points) and one entry more or less of
# a few. True residuals by the oracle at twice the tolerance asked for.
@pytest.mark.parametrize("prec", ["FP64", "MIXED"])
def test_batch_vectors_start_anywhere(torch_cuda, ib, orc, prec):
    prec = getattr(ib, prec)
    points = [(3, 3), (3, 5), (32, 64), (5, 7), (683, 3), (7, 11), (6, 3), (4, 4), (23, 89), (61, 67), (9, 9)]
    meshes = [ib.unit_square(2, m - 2, n - 2) for m, n in points]
    batch = ib.Batch(meshes, precision=prec)
    assert {int(o) % 4 for o in batch.offsets[:-1]} == {0, 1, 2, 3}
    b = splitmix_uniform(31, -1.0, 1.0, batch.ntot)
    x = torch_cuda.zeros(batch.ntot, dtype=torch_cuda.float64, device="cuda")
    st, its, _ = batch.solve(torch_cuda.from_numpy(b).cuda(), x, precision=prec, rtol=1e-10)
    assert st.converged == len(points)
    x = x.cpu().numpy()
    for i, m in enumerate(meshes):
        s, e = batch.offsets[i], batch.offsets[i + 1]
        r = b[s:e] - orc.apply_mf(m, x[s:e], sign=1.0, bc=1)
        assert np.linalg.norm(r) <= 2e-10 * np.linalg.norm(b[s:e]), points[i]
    batch.close()


# Patches of a few rows: one strip while one strip wide and three rows high (p =
# 1: four), so that a MatMult is one launch; one row or column more and it is two.
@pytest.mark.parametrize("p,nex,ney,one", [(1, 16, 4, True), (1, 12, 5, False), (1, 3, 3, True), (2, 16, 3, True),
                                           (2, 5, 4, False), (2, 17, 3, False), (3, 9, 3, True), (4, 7, 1, True),
                                           (5, 16, 1, True)])
@pytest.mark.parametrize("geom", [0, 1])
def test_patches_of_a_few_rows(torch_cuda, ib, orc, p, nex, ney, one, geom):
    M = distorted(ib.unit_square(p, nex, ney))
    x = splitmix_uniform(p * 10 + nex, -1.0, 1.0, (nex + p) * (ney + p))
    plan = ib.Plan(M, geometry=geom)
    assert (plan.info.rows_per_strip >= ney) == one
    xd = torch_cuda.from_numpy(x).cuda()
    yd = torch_cuda.full_like(xd, float("nan"))
    plan.apply(xd, yd)
    assert rel(yd.cpu().numpy(), orc.apply_mf(M, x)) < 1e-12
    plan.close()
