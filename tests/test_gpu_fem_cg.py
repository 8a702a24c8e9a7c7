"""The reference's preconditioner (inner Jacobi-CG on the bilinear FEM matrix)
where plans, options and the solver's two loops meet: plans of several sizes
alive together, iteration caps, breakdowns, waits that run out.
"""
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


def random_vector(torch, plan, seed, dtype=None):
    return torch.from_numpy(splitmix_uniform(seed, -1.0, 1.0, plan.nfunc)).to("cuda", dtype or torch.float64)


def free_vector(torch, mesh, seed):
    """Random right-hand side, zero on the boundary ring."""
    m, n = mesh["nex"] + mesh["p"], mesh["ney"] + mesh["p"]
    b = splitmix_uniform(seed, -1.0, 1.0, m * n).reshape(n, m)
    b[0], b[-1], b[:, 0], b[:, -1] = 0.0, 0.0, 0.0, 0.0
    return torch.from_numpy(b.ravel().copy()).cuda()


# Plans of several sizes in use at once: their cluster kernels are the same
# functions with different amounts of shared memory (64^2 and 32^2: four rows
# per thread, 9 KB and 3 KB; 500 x 120: above the 48 KB a function may ask for
# without a limit of its own; 3 x 1200: many rows per CTA). Each call gives the
# same bits before and after the other plans came into use.
@pytest.mark.parametrize("prec", [0, 1])
def test_plans_of_several_sizes_together(torch_cuda, ib, prec):
    torch = torch_cuda
    dt = torch.float32 if prec else torch.float64
    plans, first = [], []
    for nex, ney in [(500, 120), (64, 64), (3, 1200), (32, 32), (8, 40)]:
        plan = ib.Plan(ib.unit_square(2, nex, ney))
        r = random_vector(torch, plan, nex, dt)
        z = torch.full_like(r, float("nan"))
        plan.pc_apply(r, z, pc=ib.PC_FEM_CG, precision=prec, pc_rtol=1e-3)
        plans.append((plan, r))
        first.append(z)
    for (plan, r), z in zip(plans, first):
        z2 = torch.full_like(r, float("nan"))
        plan.pc_apply(r, z2, pc=ib.PC_FEM_CG, precision=prec, pc_rtol=1e-3)
        assert torch.equal(z, z2)
        plan.close()


# Waits that run out at once: IGA_ERR_TIMEOUT, z as it was, and the plan
# solves on as before, its loop included (sizes of 1, 8 and 16 CTAs).
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("nex,ney", [(40, 33), (20, 1), (255, 62), (3, 1200)])
def test_waits_that_run_out(torch_cuda, ib, nex, ney, prec):
    torch = torch_cuda
    mesh = ib.unit_square(1, nex, ney)
    plan = ib.Plan(mesh)
    r = random_vector(torch, plan, nex, torch.float32 if prec else torch.float64)
    z = torch.full_like(r, float("nan"))
    tol = 1e-3 if prec else 1e-10
    plan.pc_apply(r, z, pc=ib.PC_FEM_CG, precision=prec, pc_rtol=tol)
    plan.set_wait_limit(0)
    for _ in range(2):
        z2 = torch.full_like(r, 3.0)
        with pytest.raises(ib.IgaError) as e:
            plan.pc_apply(r, z2, pc=ib.PC_FEM_CG, precision=prec, pc_rtol=tol)
        assert e.value.status == 8   # IGA_ERR_TIMEOUT
        assert torch.equal(z2, torch.full_like(r, 3.0))
    for polls in (1, 2, 4, 8, 16, 64):   # some waits end in time, others run out
        plan.set_wait_limit(polls)
        for _ in range(5):
            z2 = torch.full_like(r, 3.0)
            try:
                plan.pc_apply(r, z2, pc=ib.PC_FEM_CG, precision=prec, pc_rtol=tol)
                assert torch.equal(z, z2)
            except ib.IgaError as e:
                assert e.status == 8
    plan.set_wait_limit(0)
    if not prec:
        b, x = free_vector(torch, mesh, 2), torch.zeros(plan.nfunc, dtype=torch.float64, device="cuda")
        if float(b.abs().max()) > 0.0:
            assert plan.solve(b, x, check=False, pc=ib.PC_FEM_CG, max_it=3).status != 0
        with pytest.raises(ib.IgaError):
            plan.spectrum(pc=ib.PC_FEM_CG, steps=3)
    plan.set_wait_limit(-1)
    plan.device_status()   # the MatMult's waits ran out too
    z2 = torch.full_like(r, float("nan"))
    plan.pc_apply(r, z2, pc=ib.PC_FEM_CG, precision=prec, pc_rtol=tol)
    assert torch.equal(z, z2)
    if not prec and float(b.abs().max()) > 0.0:
        assert plan.solve(b, x, pc=ib.PC_FEM_CG, max_it=50).relres <= 1e-10
    plan.close()


# No outer iteration asked for: none done, x as it was.
@pytest.mark.parametrize("prec", ["FP64", "MIXED", "MIXED_PC"])
def test_no_outer_iteration(torch_cuda, ib, prec):
    torch = torch_cuda
    mesh = ib.unit_square(2, 40, 33)
    plan = ib.Plan(mesh, precision=ib.MIXED)
    b, x0 = free_vector(torch, mesh, 4), free_vector(torch, mesh, 5)
    x = x0.clone()
    st = plan.solve(b, x, check=False, precision=getattr(ib, prec), pc=ib.PC_FEM_CG, max_it=0, x0_nonzero=1)
    assert st.status == 5 and st.iterations == 0   # IGA_ERR_NOT_CONVERGED
    assert torch.equal(x, x0)
    plan.close()


# A right-hand side whose first inner p.Kp underflows to zero (2.3e-162 squared
# over diag = 8/3 is under half the smallest double): the preconditioner breaks
# down before any outer iteration.
def test_inner_breakdown_ends_the_solve(torch_cuda, ib):
    torch = torch_cuda
    plan = ib.Plan(ib.unit_square(2, 64, 64))
    b = torch.zeros(plan.nfunc, dtype=torch.float64, device="cuda")
    b[33 * 66 + 33] = 2.3e-162
    x = torch.full_like(b, 1.0)
    st = plan.solve(b, x, check=False, pc=ib.PC_FEM_CG)
    assert st.status == 6 and st.iterations == 0   # IGA_ERR_BREAKDOWN
    assert float(x.abs().max()) == 0.0
    # and the plan solves on
    b = free_vector(torch, plan.mesh, 6)
    assert plan.solve(b, x, pc=ib.PC_FEM_CG).relres <= 1e-10
    plan.close()


# The solver's loop on the device and from the host: the same kernels in the
# same order, so the same bits, iterations and inner iterations, with every
# preconditioner and in every precision, with and without a kappa; and a
# cap that ends both loops early.
@pytest.mark.parametrize("prec", ["FP64", "MIXED", "MIXED_PC"])
@pytest.mark.parametrize("pc", ["NONE", "FEM_EXACT", "FEM_CG"])
@pytest.mark.parametrize("p,nex,ney", [(2, 40, 33), (3, 129, 70)])
def test_device_and_host_loops_agree(torch_cuda, ib, p, nex, ney, pc, prec):
    torch = torch_cuda
    mesh = ib.unit_square(p, nex, ney)
    plan = ib.Plan(mesh, precision=ib.MIXED)
    b = free_vector(torch, mesh, p)
    kappa = torch.from_numpy(splitmix_uniform(8, 0.5, 2.0, nex * ney * (p + 1) ** 2)).cuda()
    for with_kappa in (False, True):
        if with_kappa:
            plan.set_kappa(kappa)
        for max_it in (3, 40):
            got = []
            for graph in (1, 0):
                plan.set_solver_graph(graph)
                x = torch.zeros_like(b)
                st = plan.solve(b, x, check=False, precision=getattr(ib, prec), pc=getattr(ib, "PC_" + pc),
                                max_it=max_it)
                got.append((x, st.status, st.iterations, st.pc_iterations, st.sweeps, st.relres))
            assert got[0][1:] == got[1][1:]
            assert torch.equal(got[0][0], got[1][0])
    plan.close()


# An infinite entry of the boundary ring couples to no interior one: no
# breakdown, but a residual norm without meaning, so NaN everywhere, in one
# cluster (1, 8 and 16 CTAs) as past it (600 x 300: a launch per step).
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("nex,ney", [(20, 1), (40, 33), (255, 62), (600, 300)])
@pytest.mark.parametrize("where", ["corner", "side", "top"])
def test_infinity_on_the_boundary_ring(torch_cuda, ib, nex, ney, prec, where):
    torch = torch_cuda
    plan = ib.Plan(ib.unit_square(2, nex, ney))
    m, n = nex + 2, ney + 2
    r = random_vector(torch, plan, nex, torch.float32 if prec else torch.float64)
    r[{"corner": 0, "side": (n // 2) * m, "top": (n - 1) * m + m // 2}[where]] = float("-inf")
    z = torch.full_like(r, 3.0)
    plan.pc_apply(r, z, pc=ib.PC_FEM_CG, precision=prec)
    assert bool(torch.isnan(z).all())
    plan.close()


# Powers of two pass through the iteration unchanged while nothing overflows:
# entries up to 2^126 of FP32's 2^128, and well inside the rest of both ranges,
# although the mesh's stiffness factors are about 130 (64 elements) to 2000
# (1000) and its mass factors as much under 1.
@pytest.mark.parametrize("prec,k", [(1, 126), (1, -80), (0, 400), (0, -400)])
@pytest.mark.parametrize("nex,ney", [(64, 64), (3, 1000), (40, 33)])
def test_scaled_right_hand_sides(torch_cuda, ib, nex, ney, prec, k):
    torch = torch_cuda
    plan = ib.Plan(ib.unit_square(2, nex, ney))
    r = random_vector(torch, plan, nex, torch.float32 if prec else torch.float64)
    got = []
    for scale in (1.0, 2.0 ** k):
        z = torch.full_like(r, float("nan"))
        plan.pc_apply(r * scale, z, pc=ib.PC_FEM_CG, precision=prec, pc_max_it=1)
        got.append(z / scale)
    assert torch.equal(got[0], got[1])
    plan.close()


def fem_diagonal(gx, gy):
    """Diagonal of the bilinear FEM matrix on the tensor grid gx x gy, 1 on the boundary ring."""
    def factors(g):
        h = np.diff(g)
        return 1.0 / h[:-1] + 1.0 / h[1:], (h[:-1] + h[1:]) / 3.0
    (kx, mx), (ky, my) = factors(gx), factors(gy)
    d = np.ones((len(gy), len(gx)))
    d[1:-1, 1:-1] = np.outer(my, kx) + np.outer(ky, mx)
    return d.ravel()


# A cap of one inner iteration: z = alpha p with p = r / diag and alpha = r.p /
# p.Kp, in one cluster (rows per thread as above) and past it. A row of K p is
# nine terms of about one rounding each and the sums are FP64: 1e-12 and 1e-5.
@pytest.mark.parametrize("prec,tol", [(0, 1e-12), (1, 1e-5)])
@pytest.mark.parametrize("p,nex,ney", [(2, 64, 64), (3, 40, 1), (1, 2, 30), (2, 17, 90), (3, 300, 125), (2, 600, 300)])
def test_one_inner_iteration(torch_cuda, ib, orc, p, nex, ney, prec, tol):
    torch = torch_cuda
    plan = ib.Plan(ib.unit_square(p, nex, ney))
    gx, gy = plan.fem_nodes()
    rd = random_vector(torch, plan, nex + p, torch.float32 if prec else torch.float64)
    z = torch.full_like(rd, float("nan"))
    plan.pc_apply(rd, z, pc=ib.PC_FEM_CG, precision=prec, pc_rtol=1e-14, pc_max_it=1)
    r = rd.double().cpu().numpy()
    d = r / fem_diagonal(gx, gy)
    ref = (r @ d) / (d @ orc.fem_matvec(gx, gy, d)) * d
    assert np.abs(z.double().cpu().numpy() - ref).max() <= tol * np.abs(ref).max()
    plan.close()


# Inner caps and tolerances belong to the call: a plan that has solved with
# others does as many inner iterations, and gives the same bits, as one that has
# not.
@pytest.mark.parametrize("prec", ["FP64", "MIXED", "MIXED_PC"])
def test_inner_options_of_each_solve(torch_cuda, ib, prec):
    torch = torch_cuda
    mesh = ib.unit_square(2, 50, 44)
    b = free_vector(torch, mesh, 12)
    options = [dict(pc_max_it=4, pc_rtol=1e-10), dict(pc_max_it=9, pc_rtol=1e-10), dict(pc_max_it=500, pc_rtol=1e-2),
               dict(pc_max_it=500, pc_rtol=1e-4), dict(pc_max_it=4, pc_rtol=1e-10)]

    def solve(plan, kw):
        x = torch.zeros_like(b)
        st = plan.solve(b, x, check=False, precision=getattr(ib, prec), pc=ib.PC_FEM_CG, max_it=5, max_sweeps=2, **kw)
        return x, st.iterations, st.pc_iterations

    shared = ib.Plan(mesh, precision=ib.MIXED)
    counts = []
    for kw in options:
        fresh = ib.Plan(mesh, precision=ib.MIXED)
        (x, *n), (x2, *n2) = solve(shared, kw), solve(fresh, kw)
        assert n == n2 and torch.equal(x, x2)
        counts.append(n[1])
        fresh.close()
    assert len(set(counts)) == 4 and counts[0] == counts[4]
    shared.close()
