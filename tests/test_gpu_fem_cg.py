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
