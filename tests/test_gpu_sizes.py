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
