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
