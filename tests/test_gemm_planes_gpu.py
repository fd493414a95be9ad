"""Several products of inputs of their own in one launch."""

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


# every token tile with a remainder, one and two k-blocks and a ragged last one, weights of one tile and of several, splits of the
# inner range and none
@pytest.mark.parametrize("tokens", [1, 3, 16, 17, 33, 64])
@pytest.mark.parametrize("planes,width,inner", [(1, 128, 72), (4, 256, 1024), (3, 1280, 200), (4, 4096, 512)])
def test_planes_are_the_products_one_by_one(tokens, planes, width, inner):
    from rapid_llm_b200.ops import kernels

    torch.manual_seed(tokens)
    x = torch.randn(planes * tokens, inner, device=DEV).bfloat16()
    w = (torch.randn(planes, width, inner, device=DEV) * inner ** -0.5).bfloat16()
    buffer = torch.full((planes * tokens + 2, width), 7.0, dtype=torch.bfloat16, device=DEV)
    fault = torch.zeros(1, dtype=torch.int32, device=DEV)
    out = kernels.gemm_bf16_planes(x, w, buffer[1:-1], fault)
    assert int(fault) == 0 and bool((buffer[0] == 7.0).all()) and bool((buffer[-1] == 7.0).all())
    want = torch.einsum("ptk,pnk->ptn", x.view(planes, tokens, inner).double(), w.double()).view(planes * tokens, width)
    # one rounding to 8 bits of what float32 sums have left untouched at this size
    assert bool(((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all())


def test_planes_of_a_wider_tensor_are_taken_one_by_one():
    from rapid_llm_b200.ops import gemm

    torch.manual_seed(3)
    x = torch.randn(2 * 5, 256, device=DEV).bfloat16()
    wide = (torch.randn(2, 384, 256, device=DEV) / 16).bfloat16()
    fault = torch.zeros(1, dtype=torch.int32, device=DEV)
    got, want = (torch.empty(10, 256, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    gemm.planes_linear(x, wide[:, :256], got, fault)
    for plane in range(2):
        gemm.linear(x[5 * plane : 5 * plane + 5], wide[plane, :256], want[5 * plane : 5 * plane + 5], fault)
    assert int(fault) == 0 and torch.equal(got, want)
