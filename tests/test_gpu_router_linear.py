"""GPU: the router linear for many rows (tensor-core form, csrc/router.cu) against float64, at the edges of its 16 x 32 tiles
and of its blocks of 32 along d."""

import pytest
import torch

from zmlx_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("T", [9, 16, 17, 100])
@pytest.mark.parametrize("E,d", [(1, 32), (33, 64), (128, 2048), (256, 7168), (31, 288), (32, 40)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_router_linear(T, E, d, dtype):
    g = torch.Generator(device=DEV).manual_seed(T * E + d)
    x = torch.randn((T, d), generator=g, device=DEV).to(torch.bfloat16)
    w = (torch.randn((E, d), generator=g, device=DEV) * 0.02).to(torch.bfloat16)
    got = ops.router_logits(x, w, out_dtype=dtype).double()
    ref, mass = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    # d float32 additions of exact products, each within 2^-23 of the partial sum, and the result's rounding
    bound = d * 2.0 ** -23 * mass + (2.0 ** -8 * ref.abs() if dtype == torch.bfloat16 else 0.0)
    assert bool(((got - ref).abs() <= bound).all())
    assert torch.equal(got, ops.router_logits(x, w, out_dtype=dtype).double())
