"""The coefficient: the forms of array that iga_plan_set_kappa takes."""
import numpy as np
import pytest

from iga_testlib import load_binding, splitmix_uniform

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


# The array may lie anywhere a copy can reach: in pinned host memory, or on the
# device at an address that is no multiple of 8 bytes.
@pytest.mark.parametrize("geom", [0, 1])
def test_kappa_arrays_a_copy_takes(torch_cuda, ib, geom):
    torch = torch_cuda
    p, nex, ney = 3, 37, 21
    mesh = ib.unit_square(p, nex, ney)
    kq = torch.from_numpy(np.exp(splitmix_uniform(8, -1.0, 1.0, nex * ney * (p + 1) ** 2)))
    shifted = torch.empty(2 * kq.numel() + 1, dtype=torch.int32, device="cuda")[1:]
    shifted.copy_(kq.view(torch.int32))
    assert shifted.data_ptr() % 8 == 4
    r = torch.from_numpy(splitmix_uniform(9, -1.0, 1.0, (nex + p) * (ney + p))).cuda()
    got = []
    for arr in (kq.cuda(), kq.pin_memory(), shifted):
        plan = ib.Plan(mesh, geometry=geom)
        plan.set_kappa(arr)
        y, z = (torch.full_like(r, float("nan")) for _ in range(2))
        plan.apply(r, y)
        plan.pc_apply(r, z)
        got.append((y, z))
        plan.close()
    for y, z in got[1:]:
        assert torch.equal(y, got[0][0]) and torch.equal(z, got[0][1])


def support_scaling(kq, p, nex, ney):
    """1 / sqrt(mean of kappa over the quadrature points of the elements that support each control point)."""
    m, n = nex + p, ney + p
    total, count = np.zeros((n, m)), np.zeros((n, m))
    per = kq.reshape(ney, nex, -1).sum(axis=2)
    for b in range(p + 1):      # element (ey, ex) supports control points (ey + b, ex + a)
        for a in range(p + 1):
            total[b:b + ney, a:a + nex] += per
            count[b:b + ney, a:a + nex] += (p + 1) ** 2
    return 1.0 / np.sqrt(total / count)


# The kappa scaling S of the preconditioner, with a kappa that differs at every
# quadrature point: z with a kappa = S z0(S r) of a plan without one. Sizes
# below one tile of 32 x 8 control points, of exactly one (p = 3, 29 x 5), one
# more, and ragged ones in both directions. FP64: the two differ by the
# rounding of S, which the exact inverse does not raise against z's largest
# entry (1e-12 with room); FP32: four TF32 roundings of 2^-11 (two transforms,
# two operands); inner CG: twice pc_rtol = 1e-13 times a condition under 1e4.
@pytest.mark.parametrize("p,nex,ney", [(1, 1, 1), (1, 3, 2), (1, 70, 19), (2, 5, 9), (2, 95, 41), (3, 29, 5),
                                       (3, 30, 6), (4, 33, 18), (4, 6, 61), (5, 27, 30), (5, 60, 11)])
def test_scaling_of_a_varying_kappa(torch_cuda, ib, p, nex, ney):
    mesh = ib.unit_square(p, nex, ney)
    plain, plan = ib.Plan(mesh), ib.Plan(mesh)
    r = splitmix_uniform(p + nex, -1.0, 1.0, plan.nfunc)
    for seed in (1, 2):   # the second kappa replaces the first
        kq = 10.0 ** splitmix_uniform(seed + nex, -1.0, 1.0, nex * ney * (p + 1) ** 2)
        plan.set_kappa(torch_cuda.from_numpy(kq).cuda())
        S = torch_cuda.from_numpy(support_scaling(kq, p, nex, ney).ravel()).cuda()
        for prec, pc, split, tol in [(ib.FP64, ib.PC_FEM_EXACT, 1, 1e-12), (ib.FP64, ib.PC_FEM_EXACT, 0, 1e-12),
                                     (ib.FP64, ib.PC_FEM_CG, 1, 1e-8), (ib.FP32, ib.PC_FEM_EXACT, 1, 4 * 2.0 ** -11)]:
            if prec == ib.FP32 and min(plan.nfunc // (nex + p), nex + p) == 2:
                continue   # no free control points: the FP32 transforms refuse that
            dt = torch_cuda.float32 if prec == ib.FP32 else torch_cuda.float64
            rd, Sd = torch_cuda.from_numpy(r).to("cuda", dt), S.to(dt)
            z, z0 = torch_cuda.full_like(rd, float("nan")), torch_cuda.full_like(rd, float("nan"))
            for pl, src, dst in ((plan, rd, z), (plain, Sd * rd, z0)):
                pl.set_pc_split(split)
                pl.pc_apply(src, dst, pc=pc, precision=prec, pc_rtol=1e-13)
            ref = (Sd * z0).double()
            assert float((z.double() - ref).abs().max()) <= tol * float(ref.abs().max())
    plain.close()
    plan.close()


# A kappa set after a solve: the loop that the solve left behind takes the new
# scaling (the same bits as a plan that never had another one).
@pytest.mark.parametrize("prec", ["FP64", "MIXED", "MIXED_PC"])
@pytest.mark.parametrize("pc", ["FEM_EXACT", "FEM_CG"])
def test_second_kappa_in_the_solvers_loop(torch_cuda, ib, pc, prec):
    p, nex, ney = 3, 45, 38
    mesh = ib.unit_square(p, nex, ney)
    m, n = nex + p, ney + p
    b = splitmix_uniform(3, -1.0, 1.0, m * n).reshape(n, m)
    b[0], b[-1], b[:, 0], b[:, -1] = 0.0, 0.0, 0.0, 0.0
    b = torch_cuda.from_numpy(b.ravel().copy()).cuda()
    k1, k2 = [torch_cuda.from_numpy(10.0 ** splitmix_uniform(s, -1.0, 1.0, nex * ney * (p + 1) ** 2)).cuda()
              for s in (4, 5)]
    got = []
    for kappas in ([k1, k2], [k2]):
        plan = ib.Plan(mesh, precision=ib.MIXED)
        for k in kappas:
            plan.set_kappa(k)
            x = torch_cuda.zeros_like(b)
            st = plan.solve(b, x, check=False, precision=getattr(ib, prec), pc=getattr(ib, "PC_" + pc), max_it=25)
        got.append((x, st.iterations, st.pc_iterations))
        plan.close()
    assert got[0][1:] == got[1][1:] and torch_cuda.equal(got[0][0], got[1][0])
